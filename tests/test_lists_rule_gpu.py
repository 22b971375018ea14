"""Which whole graphs take the tile lists: those whose rows are nearer to their pivot than to the other
pivots, by enough for the plan to pay.  Told by the stages of the call; the graphs themselves are
compared with the full scan's."""
import ctypes as C

import numpy as np
import pytest
import torch

from evoc import _lib

pytestmark = pytest.mark.gpu


def _rows(kind, n, d, clusters, mean=0.0, spread=0.4):
    g = torch.Generator().manual_seed(n + d + clusters)
    lab = torch.randint(0, max(clusters, 1), (n,), generator=g)
    x = spread * torch.randn(n, d, generator=g) + mean * torch.randn(d, generator=g)
    if clusters:
        x += torch.randn(clusters, d, generator=g)[lab]
    if kind == "bits":
        p = torch.rand(max(clusters, 1), d, generator=g) < (0.2 if clusters > 1 else 0.5)
        flip = 0.01 if clusters > 1 else 0.1
        return np.packbits((p[lab] ^ (torch.rand(n, d, generator=g) < flip)).numpy(), axis=1)
    x = (x / x.norm(dim=1, keepdim=True)).numpy()
    return x if kind == "f32" else np.clip(np.round(127 * x), -127, 127).astype(np.int8)


def _call(x, k, rows=None):
    code = {np.dtype(np.float32): 0, np.dtype(np.int8): 1, np.dtype(np.uint8): 2}[x.dtype]
    a, b = rows or (0, len(x))
    ctx = _lib.Context(0)
    try:
        ctx.profile(True)
        ind, dst = np.empty((b - a, k), np.int32), np.empty((b - a, k), np.float32)
        o = _lib.default_opts()
        o.certify = 0
        if rows:
            o.row_begin, o.row_end = rows
        p = C.c_void_p
        st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(o), code, x.ctypes.data_as(p), len(x), x.shape[1], k, None,
                                           ind.ctypes.data_as(p), dst.ctypes.data_as(p), None)
        assert st == 0, ctx.last_error()
        return ind, dst, {s for s, _ in ctx.stages()}
    finally:
        ctx.close()


@pytest.mark.parametrize("kind,n,d,clusters,mean,lists", [
    ("f32", 18900, 96, 20, 0.0, False),     # no more query blocks than SMs
    ("f32", 24000, 96, 20, 0.0, True),
    ("f32", 24000, 96, 0, 1.0, False),      # a common mean and nothing else: every cosine about 0.86
    ("f32", 60000, 96, 0, 2.0, False),
    ("f32", 60000, 96, 50, 1.0, True),      # clusters about a common mean
    ("i8", 24000, 96, 10, 0.0, True),
    ("i8", 24000, 96, 200, 0.0, False),     # pivots in a fifth of the clusters
    ("i8", 60000, 96, 50, 0.0, True),
    ("i8", 60000, 96, 0, 1.0, False),
    ("f32", 60000, 32, 0, 0.0, False),      # few dimensions: pivots near by without clusters
    ("i8", 60000, 32, 0, 0.0, False),
    ("i8", 60000, 32, 50, 0.0, True),
    ("bits", 60000, 512, 20, 0.0, True),
    ("bits", 60000, 512, 1000, 0.0, False),
    ("bits", 60000, 512, 1, 0.0, False),    # dense rows of one prototype
])
def test_who_takes_the_lists(kind, n, d, clusters, mean, lists):
    x = _rows(kind, n, d, clusters, mean)
    ind, dst, stages = _call(x, 15)
    assert ("tile_lists" in stages) == lists
    part = _call(x, 15, (0, 1000))
    assert np.array_equal(ind[:1000], part[0]) and np.array_equal(dst[:1000].view(np.uint32), part[1].view(np.uint32))


def test_sampled_rows_that_are_pivots():
    """At 2^20 rows every sampled row is one of the pivots; that is no sign of clusters."""
    n, d, k = 1 << 20, 64, 5
    x = torch.randn(n, d, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    x = torch.clamp(torch.round(127 * x / x.norm(dim=1, keepdim=True)), -127, 127).to(torch.int8)
    ind, dst = torch.empty(n, k, dtype=torch.int32, device="cuda"), torch.empty(n, k, device="cuda")
    torch.cuda.synchronize()
    ctx = _lib.Context(0)
    try:
        o = _lib.default_opts()
        o.buffers_on_device = 1
        p = C.c_void_p
        st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(o), 1, p(x.data_ptr()), n, d, k, None, p(ind.data_ptr()),
                                           p(dst.data_ptr()), None)
        assert st == 0, ctx.last_error()
        assert ctx.list_stats() == {"tiles": 0, "all_tiles": 0}
    finally:
        ctx.close()
