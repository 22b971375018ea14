"""The tensor-core Jaccard scan's survivor bound from the keys' popcounts: rows from empty to full,
sorted so that a chunk's popcounts are alike or mixed so that one small row loosens its chunk, row
counts at the edges of chunks and tiles.  Bit for bit against the oracle."""
import numpy as np
import pytest

import evoc
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 256, 257, 700])
@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("k", [1, 12])
def test_popcounts_from_empty_to_full(n, order, k):
    r = np.random.default_rng(n + k)
    share = np.linspace(0.0, 1.0, n) if order == "sorted" else r.permutation(np.linspace(0.0, 1.0, n))
    base = r.random(200)
    x = np.packbits(base[None, :] * 0.5 + r.random((n, 200)) * 0.5 < share[:, None], axis=1)
    x[n // 2] = x[n // 3]
    ind, dst = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="exact_int"))
    oi, orr = O.exact_knn(x, k)
    assert np.array_equal(ind, oi)
    assert np.array_equal(dst.view(np.uint32), O.transform(O.DT_U8, orr).view(np.uint32))
