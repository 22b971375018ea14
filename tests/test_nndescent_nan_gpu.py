"""NN-descent over rows some of which hold a NaN: they have no nearest pivot, take part in the first cell,
and leave the other rows' graph what it is."""
import numpy as np
import pytest

import evoc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,share", [(300, 0.02), (3000, 0.01), (3000, 0.5), (3000, 1.0)])
def test_rows_without_a_pivot(n, share):
    r = np.random.default_rng(n)
    x = r.normal(size=(10, 64))[r.integers(0, 10, n)] + 0.3 * r.normal(size=(n, 64))
    x = (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
    bad = r.random(n) < share
    x[bad, 3] = np.nan
    ind, dst = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=15, form="nndescent"), np.random.RandomState(1))
    assert ind.min() >= 0 and ind.max() < n and np.array_equal(ind[:, 0], np.arange(n))
    again, _ = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=15, form="nndescent"), np.random.RandomState(1))
    assert np.array_equal(ind, again)
    good = np.nonzero(~bad)[0]
    if len(good) > n // 2:
        sims = x[good] @ x[good].T
        np.fill_diagonal(sims, 2.0)
        want = good[np.argsort(-sims, axis=1, kind="stable")[:, :15]]
        recall = np.mean([len(set(a) & set(b)) / 15 for a, b in zip(ind[good], want)])
        assert recall >= 0.95
