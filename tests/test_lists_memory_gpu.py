"""Whole graphs whose tile lists (or small form) find no room: the call takes the plain scan with the
memory that needs, and gives the same graph.  The GPU's memory is filled by an allocation of torch's;
a server is given a budget that holds the plain scan only."""
import ctypes as C
import gc

import numpy as np
import pytest
import torch

import evoc
from evoc import _lib
from evoc.serving import Server

pytestmark = pytest.mark.gpu


def _clusters(n, d, seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.randn(20, d, generator=g, device="cuda")
    x = c[torch.randint(0, 20, (n,), generator=g, device="cuda")]
    x += 0.35 * torch.randn(n, d, generator=g, device="cuda")
    return x / x.norm(dim=1, keepdim=True)


class _Call:
    """One context; device rows and outputs."""

    def __init__(self):
        self.ctx = _lib.Context(0)
        self.ctx.profile(True)

    def __call__(self, x, k, rows=None):
        a, b = rows or (0, len(x))
        ind = torch.empty(b - a, k, dtype=torch.int32, device="cuda")
        dst = torch.empty(b - a, k, device="cuda")
        o = _lib.default_opts()
        o.buffers_on_device, o.certify = 1, 0
        if rows:
            o.row_begin, o.row_end = rows
        p = C.c_void_p
        torch.cuda.synchronize()
        st = _lib.lib().evoc_gpu_knn_graph(self.ctx.h, C.byref(o), {torch.float32: 0, torch.int8: 1}[x.dtype],
                                           p(x.data_ptr()), len(x), x.shape[1], k, None, p(ind.data_ptr()),
                                           p(dst.data_ptr()), None)
        assert st == 0, self.ctx.last_error()
        return ind, dst, {s for s, _ in self.ctx.stages()}


def _fill(leave):
    gc.collect()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(free - leave, 1), dtype=torch.uint8, device="cuda")


@pytest.fixture(autouse=True)
def _nothing_held():
    """Contexts that earlier tests share hold pools of freed memory, which the driver would hand out."""
    for ctx in list(_lib._contexts.values()):
        ctx.close()
    _lib._contexts.clear()


@pytest.mark.parametrize("kind", ["f32", "i8"])
def test_no_room_for_the_lists(kind):
    n, d, k = 400000, 256, 15
    x = _clusters(n, d)
    if kind == "i8":
        x = torch.clamp(torch.round(127 * x), -127, 127).to(torch.int8)
    call = _Call()
    want = call(x, k)
    assert "tile_lists" in want[2]
    call.ctx.close()
    call = _Call()
    call(x, k, (0, n - 1))  # the buffers of the plain scan
    spare = [torch.empty(n, k, dtype=torch.int32, device="cuda"), torch.empty(n, k, device="cuda")]  # outputs
    full = _fill(100 << 20)
    del spare
    try:
        got = call(x, k)
    finally:
        del full
        torch.cuda.empty_cache()
    assert "tile_lists" not in got[2]
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    call.ctx.close()


def test_the_lists_give_way():
    """A later call that needs the room the lists of an earlier one hold."""
    n, d, k = 400000, 256, 15
    x, y = _clusters(n, d), _clusters(600000, d, 2)
    call = _Call()
    assert "tile_lists" in call(x, k)[2]
    out = call(y, k, (0, 1000))  # loads what the call below runs
    call.ctx.close()
    call = _Call()
    call(x, k)
    full = _fill(120 << 20)  # the rows of y take 690 MB, those of x gave 460; the arena holds 400
    try:
        got = call(y, k, (0, 1000))
    finally:
        del full
        torch.cuda.empty_cache()
    assert torch.equal(got[0], out[0]) and torch.equal(got[1], out[1])
    call.ctx.close()


@pytest.mark.parametrize("n,d,dtype,form", [(60000, 64, np.float32, "bf16_rerank"), (60000, 128, np.int8, "exact_int"),
                                            (4000, 64, np.int8, "exact_int"), (4000, 64, np.float32, "bf16_rerank")])
def test_a_server_short_of_budget(n, d, dtype, form):
    """The bytes a request is told to need admit it, and are those of the plain scan."""
    x = _clusters(n, d).cpu().numpy()
    if dtype == np.int8:
        x = np.clip(np.round(127 * x), -127, 127).astype(np.int8)
    o = evoc.KnnGraphOptions(n_neighbors=15, form=form)
    want = evoc.knn_graph(x, o)
    code = _lib.DTYPE_F32 if dtype == np.float32 else _lib.DTYPE_I8
    with Server(max_inflight=1) as srv:
        resident, workspace = srv.request_bytes(code, n, d, o)
    if dtype == np.int8:  # padded rows and the scan's keys, an eighth more of each
        blocks = min((n + 127) // 128, 148)
        assert workspace <= 1.125 * ((n + 255) // 256 * 256 * 128 + blocks * 256 * 15 * 8) + 1024
    with Server(max_inflight=1, budget_bytes=resident + workspace, profile=True) as srv:
        got = srv.result(srv.submit(x, o))
        st = srv.stats()
        assert st["peak_bytes"] <= st["budget_bytes"] and st["workspace_misses"] == 0
        assert "tile_lists" not in srv.stage_totals()
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
