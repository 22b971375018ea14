"""The one-pass row preparation at the edges of its tiles (32 rows, 128 columns), with rows that are
of unit length, that are not, and that are zero; rows on the host, on the device, and on the device
off the 4-byte grid.  The certified 16-bit form then reports, bit for bit, the products of the rows
divided by their serially rounded norms; the FP32 form's neighbours agree."""
import ctypes as C

import numpy as np
import pytest
import torch

import evoc
from evoc import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _product(x, y):
    """32 partial sums of fused multiply-adds (lane l: elements l, l + 32, ...), then the tree."""
    acc = np.zeros((len(y), 32), np.float32)
    for t in range(0, len(x), 32):
        w = min(32, len(x) - t)
        p = x[t:t + w].astype(np.longdouble) * y[:, t:t + w].astype(np.longdouble)  # exact
        acc[:, :w] = (p + acc[:, :w].astype(np.longdouble)).astype(np.float32)
    for o in (16, 8, 4, 2, 1):
        acc = acc + acc[:, np.arange(32) ^ o]
    return acc[:, 0]


def _device(x, k, offset):
    n, d = x.shape
    buf = torch.zeros(x.nbytes + 16, dtype=torch.uint8, device="cuda")
    buf[offset:offset + x.nbytes] = torch.from_numpy(x.view(np.uint8).reshape(-1)).cuda()
    ind = torch.empty((n, k), dtype=torch.int32, device="cuda")
    dst = torch.empty((n, k), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    o = _lib.default_opts()
    o.form, o.buffers_on_device = _lib.FORM_BF16_RERANK, 1
    ctx = _lib.context(0)
    st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(o), 0, C.c_void_p(buf.data_ptr() + offset), n, d, k, None,
                                       C.c_void_p(ind.data_ptr()), C.c_void_p(dst.data_ptr()), None)
    assert st == 0, ctx.last_error()
    return ind.cpu().numpy(), dst.cpu().numpy()


@pytest.mark.parametrize("n,d", [(31, 1), (32, 33), (33, 64), (255, 127), (256, 128), (257, 129), (300, 257), (4100, 40)])
@pytest.mark.parametrize("unit", [True, False])
def test_rows_as_prepared(n, d, unit):
    r = np.random.default_rng(n * 1000 + d)
    x = (r.normal(size=(n, d)) + r.normal(size=d)).astype(np.float32)
    x = x / np.linalg.norm(x.astype(np.float64), axis=1, keepdims=True)
    if not unit:
        x = x * r.uniform(0.1, 30.0, (n, 1))
        x[n // 2] = 0.0
    x = np.ascontiguousarray(x, np.float32)
    k = min(6, n - 1)
    y = O.prepare_float(x)
    assert np.array_equal(y, x) == unit
    ind, dst, raw = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="bf16_rerank"), return_raw=True)
    for q in range(0, n, max(1, n // 40)):
        prod = _product(y[q], y[ind[q]])
        want = np.where(prod > 0, -prod, np.finfo(np.float32).tiny)  # the cosine's raw value
        want[ind[q] == q] = -1.0
        assert np.array_equal(raw[q], want.astype(np.float32))
    exact = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="fp32"), return_raw=True)[2]
    assert np.abs(raw - exact).max() <= (d + 40) * 2.0**-24  # two orders of a sum of d products, all within 1
    for offset in (0, 4, 2):
        i2, d2 = _device(x, k, offset)
        assert np.array_equal(i2, ind) and np.array_equal(d2.view(np.uint32), dst.view(np.uint32))
    jobs = evoc.knn_graph_batch([x, x[: n // 2 + 1]], evoc.KnnGraphOptions(n_neighbors=k, form="bf16_rerank"))
    assert np.array_equal(jobs[0][0], ind)
