"""The scan's per-row sets (eight groups of slots) and heaps, each kernel variant forced through the
tuning cache at set sizes where it changes: fewer keys than groups, exactly full groups, a ragged last
group, sets in global memory on both sides of the line between the two kinds.  More rows than the small
form takes, many equal scores at the cut (ties by row index).  Against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

from evoc import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 5100
SIZES = {0: [1, 7, 8, 9, 14], 1: [15, 16, 17, 31, 37], 2: [25, 29], 3: [57, 64, 75, 81], 5: [63, 64], 14: [90, 127],
         4: [3, 129, 257, 384, 385], 10: [8, 14], 11: [30]}


def _forced(tmp_path, monkeypatch, x, code, k, keep, row_bytes, variant):
    cache = tmp_path / "tune.txt"
    mode = {0: 0, 1: 1, 2: 2}[code]
    cache.write_text(f"evoc-tune 1 mode={mode} keep={keep} row_bytes={row_bytes} log2n={int(np.log2(N))} "
                     f"variant={variant} ms=0\n")
    monkeypatch.setenv("EVOC_TUNE_CACHE", str(cache))
    ctx = _lib.Context(0)
    try:
        ind, dst, raw = np.empty((N, k), np.int32), np.empty((N, k), np.float32), np.empty((N, k), np.float32)
        o = _lib.default_opts()
        o.form = _lib.FORM_EXACT_INT
        p = C.c_void_p
        st = _lib.lib().evoc_gpu_knn_graph_raw(ctx.h, C.byref(o), code, x.ctypes.data_as(p), N, x.shape[1], k, None,
                                               ind.ctypes.data_as(p), dst.ctypes.data_as(p), raw.ctypes.data_as(p),
                                               None)
        assert st == 0, ctx.last_error()
        return ind, raw
    finally:
        ctx.close()


@pytest.mark.parametrize("variant,k", [(v, k) for v, ks in SIZES.items() for k in ks])
@pytest.mark.parametrize("kind", ["i8", "bits"])
def test_set_sizes(tmp_path, monkeypatch, variant, k, kind):
    r = np.random.default_rng(k)
    if kind == "i8":
        x = r.integers(-3, 4, size=(N, 40)).astype(np.int8)  # few distinct dots
        x[100:160] = x[3]
        code, row_bytes = 1, 128
    else:
        x = np.packbits(r.random((N, 96)) < 0.2, axis=1)
        x[100:160] = x[3]
        code, row_bytes = 2, 128
    ind, raw = _forced(tmp_path, monkeypatch, x, code, k, k, row_bytes, variant)
    for a, b in ((0, 130), (N - 60, N)):
        oi, orr = O.exact_knn(x, k, a, b)
        assert np.array_equal(ind[a:b], oi)
        assert np.array_equal(raw[a:b].view(np.uint32), orr.view(np.uint32))
