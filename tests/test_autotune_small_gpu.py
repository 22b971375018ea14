"""The autotuner beside the small form (small.cu): it is one of the forms timed where it serves, a
context tuned at a size it does not serve keeps it for the sizes it does, and a cache file says so."""
import ctypes as C

import numpy as np
import pytest

from evoc import _lib

pytestmark = pytest.mark.gpu

SMALL = 15  # what a report calls the small form


def _tune(ctx, code, form, n, d, k, path=None):
    buf = C.create_string_buffer(4096)
    st = _lib.lib().evoc_gpu_autotune(ctx.h, code, form, n, d, k, path, buf, 4096)
    assert st == 0, ctx.last_error()
    return buf.value.decode().splitlines()


def _launches(ctx, x, k, code):
    ind, dst = np.empty((len(x), k), np.int32), np.empty((len(x), k), np.float32)
    p = C.c_void_p
    o = _lib.default_opts()
    st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(o), code, x.ctypes.data_as(p), len(x), x.shape[1], k, None,
                                       ind.ctypes.data_as(p), dst.ctypes.data_as(p), None)
    assert st == 0, ctx.last_error()
    return ctx.launches(), ind


@pytest.mark.parametrize("code", [1, 2])
def test_tuned_contexts_keep_the_small_form(tmp_path, monkeypatch, code):
    k, d = 30, 64
    r = np.random.default_rng(code)
    x = r.integers(-127, 128, size=(4500, d)).astype(np.int8) if code == 1 else r.integers(0, 256, size=(4500, d // 8),
                                                                                          dtype=np.uint8)
    plain = _lib.Context(0)
    want = _launches(plain, x, k, code)
    tuned = _lib.Context(0)
    cache = str(tmp_path / "tune.txt").encode()
    lines = _tune(tuned, code, _lib.FORM_EXACT_INT, 8000, x.shape[1], k, cache)  # the same power of two
    assert not any(ln.split()[0] == str(SMALL) for ln in lines)
    got = _launches(tuned, x, k, code)
    assert got[0] == want[0] and np.array_equal(got[1], want[1])
    monkeypatch.setenv("EVOC_TUNE_CACHE", cache.decode())
    loaded = _lib.Context(0)
    got = _launches(loaded, x, k, code)
    assert got[0] == want[0] and np.array_equal(got[1], want[1])
    for c in (plain, tuned, loaded):
        c.close()


def test_the_small_form_is_timed(tmp_path):
    ctx = _lib.Context(0)
    lines = _tune(ctx, 1, _lib.FORM_EXACT_INT, 3000, 64, 30, str(tmp_path / "tune.txt").encode())
    ms = {int(ln.split()[0]): float(ln.split()[1]) for ln in lines if not ln.startswith("chosen")}
    chosen = int(lines[-1].split("variant=")[1].split()[0])
    assert SMALL in ms and ms[chosen] <= ms[SMALL]
    ctx.close()
