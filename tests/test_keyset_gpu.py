"""The scan's per-row key sets (eight groups of slots) at the set sizes where the groups change:
fewer keys than groups, exactly full groups, a ragged last group; more rows kept than there are;
ties by row index.  Against the oracle's exact selection, bit for bit (int8)."""
import numpy as np
import pytest

import evoc
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 15, 16, 17, 31, 57, 64, 100])
def test_key_set_sizes(k):
    r = np.random.default_rng(k)
    x = r.integers(-3, 4, size=(700, 40)).astype(np.int8)  # few distinct dots: many ties at the cut
    x[100:160] = x[3]
    ind, _, raw = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="exact_int"), return_raw=True)
    oi, orr = O.exact_knn(x, k)
    assert np.array_equal(ind, oi)
    assert np.array_equal(raw.view(np.uint32), orr.view(np.uint32))


@pytest.mark.parametrize("n,k", [(9, 8), (40, 30), (129, 128)])
def test_key_set_nearly_all_rows(n, k):
    x = np.random.default_rng(n).integers(-127, 128, size=(n, 33)).astype(np.int8)
    ind, _ = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="exact_int"))
    assert np.array_equal(ind, O.exact_knn(x, k)[0])
