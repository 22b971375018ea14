"""The FP32 rerank's two forms (candidate rows through registers, or through shared memory by bulk
copies) on either side of the row lengths where the second begins (a stride of 512) and ends, which the
number of candidates decides: two rows and the keys of 16 warps no longer fit from a stride of 1,152 with
up to 64 candidates, 1,104 with up to 128 and 1,024 with more.  Every reported product is the same
sequence of fused multiply-adds, bit for bit."""
import numpy as np
import pytest

import evoc
from test_rerank_gpu import _product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,lengths", [(15, (496, 497, 512, 640, 641, 656, 752, 769, 1136, 1137)),
                                       (30, (1088, 1089)), (60, (1008, 1009))])
def test_lines_between_the_forms(k, lengths):
    n = 400
    for d in lengths:
        r = np.random.default_rng(d * 100 + k)
        x = r.normal(size=(n, d)) + 2.0 * r.normal(size=d)
        x = (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
        assert np.all(np.abs(np.sqrt((x.astype(np.float64) ** 2).sum(1)) - 1) < 1e-6)
        ind, _, raw = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="bf16_rerank", certify=False),
                                     return_raw=True)
        for q in range(0, n, 41):
            want = -_product(x[q], x[ind[q]])
            want[ind[q] == q] = -1.0
            assert np.array_equal(raw[q].view(np.uint32), want.astype(np.float32).view(np.uint32)), d
