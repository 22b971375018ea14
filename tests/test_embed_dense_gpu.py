"""The reproducible epoch over graphs whose rows are mostly long: a CTA takes such a row in tiles of 384
edges (256 and 128 for wider rows), and the launch has all the CTAs there is room for.  Rows on either
side of one and two tiles and of the line to a CTA each; bit for bit against the oracle."""
import numpy as np
import pytest

import evoc
from oracle import label_prop as L
from test_label_prop_gpu import _oracle_rng, _same_state, _tuple

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncomp", [2, 5, 8, 9, 16, 20])
def test_dense_rows(ncomp):
    n = 1300
    rng = np.random.default_rng(ncomp)
    d = rng.integers(130, 300, n)
    edges = [127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 512, 513, 767, 768, 769, 1152, 1153]
    d[rng.choice(n, len(edges), replace=False)] = edges
    indptr = np.concatenate([[0], np.cumsum(d)]).astype(np.int64)
    m = int(indptr[-1])
    assert m > 128 * n
    g = L.Csr(indptr, rng.integers(0, n, m).astype(np.int32), (0.05 + 0.95 * rng.random(m)).astype(np.float32), (n, n))
    rs = np.random.RandomState(ncomp)
    orng = _oracle_rng(rs)
    emb = evoc.node_embedding(_tuple(g), ncomp, 4, None, 0.1, 1.0, 0.5, rs)
    want = L.node_embedding(g, ncomp, 4, None, 0.1, 1.0, 0.5, orng)
    assert np.array_equal(emb.view(np.uint32), want.view(np.uint32))
    assert _same_state(rs, orng)
