"""A context gives all its device memory back when it is destroyed, whatever its calls grew."""
import ctypes as C

import numpy as np
import pytest
import torch

from evoc import _lib

pytestmark = pytest.mark.gpu


def _calls(x):
    ctx = _lib.Context(0)
    n, d = x.shape
    ind, dst = np.empty((n, 15), np.int32), np.empty((n, 15), np.float32)
    p = C.c_void_p
    for symmetric, form in ((0, _lib.FORM_BF16_RERANK), (1, _lib.FORM_BF16_RERANK), (0, _lib.FORM_NNDESCENT)):
        ctx.set_symmetric_scan(symmetric)
        o = _lib.default_opts()
        o.form = form
        st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(o), 0, x.ctypes.data_as(p), n, d, 15, None,
                                           ind.ctypes.data_as(p), dst.ctypes.data_as(p), None)
        assert st == 0, ctx.last_error()
        if symmetric:
            assert ctx.symmetric_stats()["sample_rows"] > 0
    ctx.close()


def test_destroyed_contexts_hold_nothing():
    r = np.random.default_rng(1)
    n, d = 60000, 64
    x = r.normal(size=(20, d))[r.integers(0, 20, n)] + 0.3 * r.normal(size=(n, d))
    x = (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
    _calls(x)  # loads the kernels
    torch.cuda.synchronize()
    before, _ = torch.cuda.mem_get_info()
    for _ in range(3):
        _calls(x)
    after, _ = torch.cuda.mem_get_info()
    assert before - after < 16 << 20  # the symmetric scan's arena alone is larger
