"""Sets of at most 5,000 rows, whose scores are written out and selected from (small.cu): row counts
at the edges of its list, of tiles and of its range, every row kept, and data whose scores tie so
often that the cut is searched over whole rows.  int8 and binary against the oracle bit for bit, f32
against a scan variant forced through the tuning cache."""
import ctypes as C

import numpy as np
import pytest

import evoc
from evoc import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(2, 1), (31, 30), (129, 15), (1024, 9), (1025, 100), (3000, 15), (4999, 40), (5000, 256),
                                 (5001, 15), (256, 4), (257, 4), (3500, 5), (3501, 5)])
@pytest.mark.parametrize("ties", [False, True])
def test_integer_sets(n, k, ties):
    r = np.random.default_rng(n * 3 + k)
    x = r.integers(-1, 2, size=(n, 6)).astype(np.int8) if ties else r.integers(-127, 128, size=(n, 70)).astype(np.int8)
    rows = slice(0, min(n, 300))
    ind, _, raw = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, form="exact_int"), return_raw=True)
    oi, orr = O.exact_knn(x, min(k, n - 1), 0, rows.stop)
    assert np.array_equal(ind[rows], oi) and np.array_equal(raw[rows].view(np.uint32), orr.view(np.uint32))
    b = np.packbits(r.random((n, 12 if ties else 300)) < 0.2, axis=1)
    ind, _, raw = evoc.knn_graph(b, evoc.KnnGraphOptions(n_neighbors=k, form="exact_int"), return_raw=True)
    oi, orr = O.exact_knn(b, min(k, n - 1), 0, rows.stop)
    assert np.array_equal(ind[rows], oi) and np.array_equal(raw[rows].view(np.uint32), orr.view(np.uint32))


@pytest.mark.parametrize("n,d,k,scan_type", [(40, 24, 39, 0), (1500, 96, 15, 0), (4111, 200, 30, 0), (5000, 64, 100, 1)])
def test_f32_equals_scan(tmp_path, monkeypatch, n, d, k, scan_type):
    r = np.random.default_rng(n)
    x = r.normal(size=(9, d))[r.integers(0, 9, n)] + 0.4 * r.normal(size=(n, d))
    x[r.integers(0, n, n // 10)] = x[1]
    x = (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
    o = evoc.KnnGraphOptions(n_neighbors=k, form="bf16_rerank", scan_type=["fp16", "bf16"][scan_type])
    ind, dst = evoc.knn_graph(x, o)
    keep = min(n, (5 * k + 1) // 2)
    cache = tmp_path / "tune.txt"
    cache.write_text(f"evoc-tune 1 mode=0 keep={keep} row_bytes={(d + 63) // 64 * 128} log2n={int(np.log2(n))} "
                     f"variant={3 if keep < 60 else 14 if keep < 120 else 4} ms=0\n")
    monkeypatch.setenv("EVOC_TUNE_CACHE", str(cache))
    ctx = _lib.Context(0)
    try:
        i2, d2 = np.empty_like(ind), np.empty_like(dst)
        opts = _lib.default_opts()
        opts.form, opts.scan_type = _lib.FORM_BF16_RERANK, scan_type
        P = C.c_void_p
        st = _lib.lib().evoc_gpu_knn_graph(ctx.h, C.byref(opts), 0, x.ctypes.data_as(P), n, d, k, None,
                                           i2.ctypes.data_as(P), d2.ctypes.data_as(P), None)
        assert st == 0, ctx.last_error()
    finally:
        ctx.close()
    assert np.array_equal(ind, i2) and np.array_equal(dst.view(np.uint32), d2.view(np.uint32))
