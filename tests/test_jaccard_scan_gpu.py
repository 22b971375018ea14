"""The tensor-core Jaccard scan's survivor bound from the keys' smallest popcounts, at more rows than the
small form takes: rows from empty to full, sorted so that a chunk's popcounts are alike or mixed so that
one small row loosens its chunk, row counts at the edges of chunks and tiles, copies.  Bit for bit
against the oracle, rows of all popcounts."""
import numpy as np
import pytest

import evoc
from evoc import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5001, 5024, 5025, 5120, 5121])
@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("k", [2, 12, 40])
def test_popcounts_from_empty_to_full(n, order, k):
    r = np.random.default_rng(n + k)
    share = np.linspace(0.0, 1.0, n) if order == "sorted" else r.permutation(np.linspace(0.0, 1.0, n))
    base = r.random(200)
    x = np.packbits(base[None, :] * 0.5 + r.random((n, 200)) * 0.5 < share[:, None], axis=1)
    x[n // 2] = x[n // 3]
    x[::97] = x[5]
    ind, dst, raw = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="exact_int"), return_raw=True)
    assert _lib.context(0).launches() == 4  # popcounts, expansion, smallest popcounts, one scan
    for a in (0, n // 3 - 20, n // 2 - 20, n - 60):
        oi, orr = O.exact_knn(x, k, a, a + 60)
        assert np.array_equal(ind[a:a + 60], oi)
        assert np.array_equal(raw[a:a + 60].view(np.uint32), orr.view(np.uint32))
        assert np.array_equal(dst[a:a + 60].view(np.uint32), O.transform(O.DT_U8, orr).view(np.uint32))
