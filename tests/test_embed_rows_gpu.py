"""The reproducible epoch where its division of the rows changes: one row to a warp and several, rows
beyond the fixed ones taken from the counter, the three widths of a row's lanes, and rows on either
side of the line to a CTA each; bit for bit against the oracle."""
import numpy as np
import pytest

import evoc
from oracle import label_prop as L
from test_label_prop_gpu import _oracle_rng, _same_state, _tuple

pytestmark = pytest.mark.gpu


def _random_graph(n, deg, long_rows, seed):
    rng = np.random.default_rng(seed)
    d = rng.integers(0, 2 * deg + 1, n)
    d[rng.choice(n, len(long_rows), replace=False)] = long_rows
    indptr = np.concatenate([[0], np.cumsum(d)]).astype(np.int64)
    m = int(indptr[-1])
    return L.Csr(indptr, rng.integers(0, n, m).astype(np.int32), (0.05 + 0.95 * rng.random(m)).astype(np.float32),
                 (n, n))


@pytest.mark.parametrize("n,ncomp,epochs", [
    (1, 2, 3), (33, 8, 5), (1025, 3, 4),   # one block, two
    (45000, 5, 3),                         # two rows to a warp
    (45000, 12, 2), (12000, 20, 3),        # beyond the fixed rows of 2,368 and 1,184 warps
    (320000, 3, 2),                        # beyond the fixed rows at four to a warp
])
def test_epochs_over_row_divisions(n, ncomp, epochs):
    g = _random_graph(n, 6, [127, 128, 129, 511, 512, 513] if n > 1000 else [], n + ncomp)
    rs = np.random.RandomState(n % 1000)
    orng = _oracle_rng(rs)
    emb = evoc.node_embedding(_tuple(g), ncomp, epochs, None, 0.1, 1.0, 0.5, rs)
    want = L.node_embedding(g, ncomp, epochs, None, 0.1, 1.0, 0.5, orng)
    assert np.array_equal(emb.view(np.uint32), want.view(np.uint32))
    assert _same_state(rs, orng)
