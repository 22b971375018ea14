"""The FP32 rerank's two forms (candidate rows through registers, or through shared memory by bulk
copies for 512 to 1,600 features) at the row lengths and candidate counts where they change over:
every reported product is the same sequence of fused multiply-adds, bit for bit."""
import numpy as np
import pytest

import evoc

pytestmark = pytest.mark.gpu


def _product(x, y):
    """32 partial sums of fused multiply-adds (lane l: elements l, l + 32, ...), then the tree."""
    d = len(x)
    acc = np.zeros((len(y), 32), np.float32)
    for t in range(0, d, 32):
        w = min(32, d - t)
        p = x[t:t + w].astype(np.longdouble) * y[:, t:t + w].astype(np.longdouble)  # exact
        acc[:, :w] = (p + acc[:, :w].astype(np.longdouble)).astype(np.float32)
    for o in (16, 8, 4, 2, 1):
        acc = acc + acc[:, np.arange(32) ^ o]
    return acc[:, 0]


@pytest.mark.parametrize("d", [33, 500, 512, 513, 768, 1100, 1600, 1601, 1700])
@pytest.mark.parametrize("k", [1, 13, 30, 51])
def test_products_bit_for_bit(d, k):
    r = np.random.default_rng(d * 100 + k)
    n = 300
    x = r.normal(size=(n, d)) + 2.0 * r.normal(size=d)
    x = (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
    ind, _, raw = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="bf16_rerank"), return_raw=True)
    # rows as the library renormalises them: unchanged when every norm is within 1e-5 of one
    assert np.all(np.abs(np.sqrt((x.astype(np.float64) ** 2).sum(1)) - 1) < 1e-6)
    for q in range(0, n, 23):
        want = -_product(x[q], x[ind[q]])
        want[ind[q] == q] = -1.0
        assert np.array_equal(raw[q].view(np.uint32), want.astype(np.float32).view(np.uint32))
