"""Rows that hold a NaN in the small form (small.cu): their scores are never kept, as in the scan.
Without the certificate, whose rescans would decide such rows, the two forms agree bit for bit; the
scan is forced through the tuning cache."""
import ctypes as C

import numpy as np
import pytest

from evoc import _lib

pytestmark = pytest.mark.gpu


def _graph(x, k, env, monkeypatch):
    monkeypatch.setenv("EVOC_TUNE_CACHE", env)
    ctx = _lib.Context(0)
    try:
        n, d = x.shape
        ind, dst = np.empty((n, k), np.int32), np.empty((n, k), np.float32)
        o = _lib.default_opts()
        o.form, o.certify = _lib.FORM_BF16_RERANK, 0
        p = C.c_void_p
        st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(o), 0, x.ctypes.data_as(p), n, d, k, None,
                                           ind.ctypes.data_as(p), dst.ctypes.data_as(p), None)
        assert st == 0, ctx.last_error()
        return ind, dst
    finally:
        ctx.close()


@pytest.mark.parametrize("n,k", [(40, 15), (256, 15), (300, 15), (2000, 15), (2000, 60), (4999, 30)])
@pytest.mark.parametrize("share", [0.01, 0.5, 0.995])
def test_nan_rows_as_in_the_scan(tmp_path, monkeypatch, n, k, share):
    d = 64
    r = np.random.default_rng(n + k)
    x = r.normal(size=(9, d))[r.integers(0, 9, n)] + 0.4 * r.normal(size=(n, d))
    x = (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
    x[r.random(n) < share, 3] = np.nan
    keep = min(n, (5 * k + 1) // 2)
    cache = tmp_path / "tune.txt"
    cache.write_text(f"evoc-tune 1 mode=0 keep={keep} row_bytes=128 log2n={int(np.log2(n))} "
                     f"variant={3 if keep < 60 else 4} ms=0\n")
    small = _graph(x, k, str(tmp_path / "none.txt"), monkeypatch)
    scan = _graph(x, k, str(cache), monkeypatch)
    assert np.array_equal(small[0], scan[0])
    assert np.array_equal(small[1].view(np.uint32), scan[1].view(np.uint32))
