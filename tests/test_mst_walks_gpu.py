"""The MST's warp walks and subtrees where they change: the spans of a leaf and of a block's subtree,
the widths of the neighbour lists and of the padded points, and rounds on either side of the line
between a warp for 32 points and a warp for one.  Tolerances are test_mst_gpu's (f32 sums in one order)."""
import numpy as np
import pytest

import evoc
from oracle import mst
from test_mst_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,min_samples,clusters", [
    (31, 5, 4, 1), (32, 4, 2, 1), (33, 7, 6, 1),            # one leaf, two leaves
    (2048, 8, 7, 3), (2049, 6, 8, 3), (4099, 16, 15, 3),    # one subtree, a level above it; lists of 8, 9, 16
    (1025, 17, 16, 2), (2050, 31, 31, 2),                   # subtrees of 1,024; lists of 17 and 32
    (90000, 3, 0, 2), (60000, 9, 5, 2),                     # few large components: shared walks in the last rounds
])
def test_edges_of_the_walks(n, dim, min_samples, clusters):
    rng = np.random.default_rng(n)
    c = rng.normal(size=(clusters, dim)) * 5
    x = (c[rng.integers(0, clusters, n)] + 0.3 * rng.normal(size=(n, dim))).astype(np.float32)
    edges, core = evoc.parallel_boruvka(x, min_samples, return_core=True)
    oe, oc, _ = mst.boruvka_mst(x, min_samples=min_samples)
    _check(x, edges, core, min_samples, oe, oc)


def test_all_points_equal():
    x = np.full((700, 6), 0.25, np.float32)
    edges, core = evoc.parallel_boruvka(x, 5, return_core=True)
    assert np.all(core == 0.0) and np.all(edges[:, 2] == 0.0)
    _check(x, edges, core, 5)
