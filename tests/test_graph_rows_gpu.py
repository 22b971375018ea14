"""Fuzzy-graph kernels at the edges of their forms: row counts around the 128-row tile and the
4,096-count stretch of the prefix sum, neighbour counts around the shared-memory form's 64, buckets
around the 32- and 64-entry register sorts, rows with no positive distance, missing neighbours, and
columns listed twice.  Sigma and rho against the oracle, the union
against a host merge: the same pattern, weights within the exponential's 1e-5."""
import numpy as np
import pytest

import evoc
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _union(ind, dst, sigma, rho, symmetrize):
    """Rows merged by two pointers: equal columns of a row pair up in order.  (The oracle adds up a
    column listed twice, which the engine never did; without repeats the two are the same.)"""
    n = len(ind)
    f = np.float32
    with np.errstate(over="ignore", under="ignore"):
        dr = dst - rho[:, None]
        w = np.where((dr <= 0) | (sigma[:, None] == 0), f(1), np.exp(-(dr / sigma[:, None])))
    w[(ind == -1) | (ind == np.arange(n)[:, None])] = 0.0
    rows = [sorted(((int(c), v) for c, v in zip(ind[i], w[i]) if v != 0), key=lambda e: e[0]) for i in range(n)]
    cols = [[] for _ in range(n)]
    for i, row in enumerate(rows):
        for c, v in row:
            cols[c].append((i, v))
    ip, ix, dv = [0], [], []
    for a, b in zip(rows, cols):
        b = sorted(b) if symmetrize else []
        ja = jb = 0
        while ja < len(a) or jb < len(b):
            col = min(a[ja][0] if ja < len(a) else n, b[jb][0] if jb < len(b) else n)
            ha, hb = ja < len(a) and a[ja][0] == col, jb < len(b) and b[jb][0] == col
            va, vb = a[ja][1] if ha else f(0), b[jb][1] if hb else f(0)
            ix.append(col)
            dv.append(f(va + vb) - f(va * vb if ha and hb else 0))
            ja, jb = ja + ha, jb + hb
        ip.append(len(ix))
    return np.array(ip), np.array(ix), np.array(dv, f)


def _compare(ind, dst, kf, symmetrize):
    ip, ix, dv, s, r = evoc.neighbor_graph_csr(kf, ind, dst, symmetrize)
    os_, or_ = O.fuzzy_graph(ind, dst, kf, symmetrize)[3:]
    assert np.array_equal(r, or_) and np.abs(s - os_).max() <= 1e-6 * max(1.0, np.abs(os_).max())
    oip, oix, odv = _union(ind, dst, os_, or_, symmetrize)
    assert np.array_equal(ip, oip) and np.array_equal(ix, oix)
    assert np.all(np.abs(dv - odv) <= 1e-5 * np.maximum(np.abs(odv), 1e-30))


@pytest.mark.parametrize("n,k", [(1, 1), (2, 1), (127, 5), (128, 31), (129, 33), (300, 64), (300, 65), (4095, 6),
                                 (4096, 2), (8193, 15)])
@pytest.mark.parametrize("hub", [0, 32, 33, 64, 65])
def test_rows_and_buckets(n, k, hub):
    r = np.random.default_rng(n * 7 + k + hub)
    ind = np.argsort(r.random((n, min(4 * k + 8, n))), axis=1)[:, :k] if n < 400 else r.integers(0, n, (n, k))
    ind = np.resize(ind, (n, k)).astype(np.int32)
    for i in range(min(hub, n)):  # row 0 is listed by `hub` rows
        if 0 not in ind[i]:
            ind[i, k - 1] = 0
    dst = np.sort(r.random((n, k)).astype(np.float32), axis=1)
    dst[:, 0] = 0.0
    for i in range(n):  # a column listed twice: the same distance both times
        first = {}
        for j in range(k):
            dst[i, j] = first.setdefault(int(ind[i, j]), dst[i, j])
    dst[:: 17] = 0.0
    ind[3::11, k // 2] = -1
    _compare(ind, dst, max(2.0, float(k)), True)
    if hub == 0:
        _compare(ind, dst, max(2.0, float(k)), False)
