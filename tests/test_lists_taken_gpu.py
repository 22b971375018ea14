"""Whole graphs that do take the tile lists (prune.cu), told by the stages of the call, against the
full scan (row slices) bit for bit: clusters the pivots cover, with exact copies, zero rows, rows
pointing the other way and rows of clusters too small for a pivot among them."""
import ctypes as C

import numpy as np
import pytest

from evoc import _lib

pytestmark = pytest.mark.gpu

ROWS = 40000  # above the smallest whole graph over lists, whatever the type and k


def graph(x, k, form=_lib.FORM_AUTO, rows=None, scan_type=0, certify=1):
    """(indices, distances, raw, stage names) of one call on a context of its own."""
    code = {np.dtype(np.float32): 0, np.dtype(np.int8): 1, np.dtype(np.uint8): 2}[x.dtype]
    n, d = x.shape
    a, b = rows or (0, n)
    ctx = _lib.Context(0)
    try:
        ctx.profile(True)
        ind, dst, raw = (np.empty((b - a, k), t) for t in (np.int32, np.float32, np.float32))
        o = _lib.default_opts()
        o.form, o.scan_type, o.certify = form, scan_type, certify
        if rows:
            o.row_begin, o.row_end = rows
        p = C.c_void_p
        st = _lib.lib().evoc_gpu_knn_graph_raw(ctx.h, C.byref(o), code, x.ctypes.data_as(p), n, d, k, None,
                                               ind.ctypes.data_as(p), dst.ctypes.data_as(p), raw.ctypes.data_as(p),
                                               None)
        assert st == 0, ctx.last_error()
        return ind, dst, raw, {s for s, _ in ctx.stages()}
    finally:
        ctx.close()


def same_as_slices(x, k, **opts):
    n = len(x)
    whole = graph(x, k, **opts)
    assert "tile_lists" in whole[3]
    cut = (n // 2) // 128 * 128 + 1
    for a, b in ((0, cut), (cut, n)):
        part = graph(x, k, rows=(a, b), **opts)
        assert "tile_lists" not in part[3]
        for w, p in zip(whole[:3], part[:3]):
            assert np.array_equal(w[a:b].view(np.uint32), p.view(np.uint32))


def clusters(n, d, seed, spread=0.35):
    r = np.random.default_rng(seed)
    x = r.normal(size=(20, d))[r.integers(0, 20, n)] + spread * r.normal(size=(n, d))
    few = r.permutation(n)[: n // 20]  # clusters of 25 rows
    x[few] = r.normal(size=(len(few) // 25 + 1, d))[np.arange(len(few)) // 25] + spread * r.normal(size=(len(few), d))
    x = (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
    x[r.integers(0, n, n // 20)] = x[5]
    x[r.integers(0, n, 50)] = 0.0
    x[r.integers(0, n, n // 30)] *= -1.0
    return x


def bit_clusters(n, nbytes, seed, flip=0.01):
    r = np.random.default_rng(seed)
    protos = r.random((20, nbytes * 8)) < 0.2
    rows = protos[r.integers(0, 20, n)] ^ (r.random((n, nbytes * 8)) < flip)
    rows[r.integers(0, n, n // 20)] = rows[7]
    rows[r.integers(0, n, 40)] = False
    rows[r.integers(0, n, 40)] = True
    return np.packbits(rows, axis=1)


@pytest.mark.parametrize("n,nbytes,k", [(ROWS, 16, 15), (ROWS + 129, 33, 7), (ROWS + 255, 128, 30), (ROWS, 64, 1)])
def test_bits(n, nbytes, k):
    same_as_slices(bit_clusters(n, nbytes, n + k), k, form=_lib.FORM_EXACT_INT)


@pytest.mark.parametrize("n,d,k", [(ROWS, 128, 15), (ROWS + 255, 50, 20), (ROWS + 1, 300, 40)])
def test_int8(n, d, k):
    x = np.clip(np.round(127 * clusters(n, d, n + k)), -127, 127).astype(np.int8)
    same_as_slices(x, k, form=_lib.FORM_EXACT_INT)


@pytest.mark.parametrize("n,d,k,scan_type", [(ROWS, 64, 15, 0), (ROWS + 1, 200, 30, 1), (ROWS + 127, 96, 9, 0)])
def test_f32(n, d, k, scan_type):
    # without the certificate: what the rescans of failed rows do depends on how many a call has
    same_as_slices(clusters(n, d, n + k), k, form=_lib.FORM_BF16_RERANK, scan_type=scan_type, certify=0)
