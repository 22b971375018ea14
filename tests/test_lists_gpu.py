"""Whole-graph requests over tile lists (prune.cu) against the full scan on the GPU.

A row slice takes the full scan, a whole graph of 16,384 rows or more the lists; the lists skip
only key tiles that provably hold no neighbour, so the two must agree bit for bit, whatever the
data: clusters of any size and order, none at all, duplicates (ties by row index), zero rows, rows
pointing away from each other, row counts at the edges of tiles and groups.
"""
import numpy as np
import pytest

import evoc

pytestmark = pytest.mark.gpu

MIN_ROWS = 16384  # smallest whole graph that takes the lists


def _clustered(n, d, clusters, spread, seed):
    r = np.random.default_rng(seed)
    x = r.normal(size=(clusters, d))[r.integers(0, clusters, n)] + spread * r.normal(size=(n, d))
    return (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)


def _unlike(n, d, seed):
    """Rows the bound has no easy case for: tiny clusters, exact copies, zero rows, opposite rows."""
    x = _clustered(n, d, max(2, n // 40), 0.5, seed)
    r = np.random.default_rng(seed + 1)
    x[r.integers(0, n, n // 8)] = x[5]
    x[r.integers(0, n, 50)] = 0.0
    x[r.integers(0, n, n // 10)] *= -1.0
    return x


def _same_as_slices(x, k, **opts):
    n = len(x)
    o = evoc.KnnGraphOptions(n_neighbors=k, **opts)
    whole = evoc.knn_graph(x, o, return_raw=True)
    cut = (n // 2) // 128 * 128
    for a, b in ((0, cut), (cut, n)):
        part = evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=k, row_begin=a, row_end=b, **opts), return_raw=True)
        for w, p in zip(whole, part):
            assert np.array_equal(w[a:b].view(np.uint32), p.view(np.uint32))


@pytest.mark.parametrize("scan_type", ["fp16", "bf16"])
@pytest.mark.parametrize("n,d,k", [(MIN_ROWS, 64, 15), (MIN_ROWS + 1, 200, 30), (20011, 96, 5)])
def test_f32_lists_equal_full_scan(n, d, k, scan_type):
    _same_as_slices(_clustered(n, d, 30, 0.4, 1), k, form="bf16_rerank", scan_type=scan_type)
    _same_as_slices(_clustered(n, d, 1, 1.0, 2), k, form="bf16_rerank", scan_type=scan_type)


def test_f32_lists_unlike_rows():
    _same_as_slices(_unlike(17000, 80, 3), 10, form="bf16_rerank")


@pytest.mark.parametrize("n,d,k", [(MIN_ROWS, 128, 15), (MIN_ROWS + 255, 50, 1), (18000, 300, 40)])
def test_int8_lists_equal_full_scan(n, d, k):
    for x in (_clustered(n, d, 25, 0.3, 4), _unlike(n, d, 5)):
        _same_as_slices(np.clip(np.round(127 * x), -127, 127).astype(np.int8), k, form="exact_int")


@pytest.mark.parametrize("n,nbytes,k", [(MIN_ROWS, 16, 15), (MIN_ROWS + 129, 33, 7), (20000, 128, 30)])
def test_bit_lists_equal_full_scan(n, nbytes, k):
    r = np.random.default_rng(6)
    protos = r.random((60, nbytes * 8)) < 0.1
    rows = protos[r.integers(0, 60, n)] ^ (r.random((n, nbytes * 8)) < 0.04)
    rows[:300] = rows[7]
    rows[r.integers(0, n, 40)] = False
    _same_as_slices(np.packbits(rows, axis=1), k, form="exact_int")
    _same_as_slices(np.packbits(r.random((n, nbytes * 8)) < 0.3, axis=1), k, form="exact_int")
