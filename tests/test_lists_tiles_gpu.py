"""The tiles a scan over lists reports: fewer than the full scan's where clusters are apart, all of them
in one group of all rows, none where no lists are taken."""
import ctypes as C

import numpy as np
import pytest

from evoc import _lib
from test_lists_taken_gpu import clusters

pytestmark = pytest.mark.gpu


def _stats(x, k=15, rows=None):
    ctx = _lib.Context(0)
    try:
        a, b = rows or (0, len(x))
        ind, dst = np.empty((b - a, k), np.int32), np.empty((b - a, k), np.float32)
        o = _lib.default_opts()
        if rows:
            o.row_begin, o.row_end = rows
        p = C.c_void_p
        st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(o), 1, x.ctypes.data_as(p), len(x), x.shape[1], k, None,
                                           ind.ctypes.data_as(p), dst.ctypes.data_as(p), None)
        assert st == 0, ctx.last_error()
        return ctx.list_stats()
    finally:
        ctx.close()


def test_tiles(monkeypatch):
    n = 40000  # 313 blocks of rows, 157 tiles
    x = np.clip(np.round(127 * clusters(n, 96, 3)), -127, 127).astype(np.int8)
    st = _stats(x)
    assert st["all_tiles"] == 313 * 157 and 313 <= st["tiles"] < 0.7 * st["all_tiles"]
    assert _stats(x, rows=(0, n - 1)) == {"tiles": 0, "all_tiles": 0}
    assert _stats(x[:10000]) == {"tiles": 0, "all_tiles": 0}
    monkeypatch.setenv("EVOC_LIST_LIMITS", "1,1")
    st = _stats(x)
    assert st["tiles"] == 313 * 256  # one group of 256 tiles, 99 past the data
