"""The tile lists' bound, restated in NumPy: for any two groups of rows and any two centres the
largest product between their rows never exceeds it, and the binary form never understates J.
(The kernels of prune.cu compute it; tests/test_lists_gpu.py compares whole graphs.)"""
import numpy as np
import pytest


def _stats(x, m):
    mm = float(m @ m)
    a = (x @ m) / mm if mm > 0 else np.zeros(len(x))
    rho = np.sqrt(np.maximum((x * x).sum(1) - a * a * mm, 0.0))
    return a, rho.max()


def _bound(x, y, mx, my):
    a, ra = _stats(x, mx)
    c, rc = _stats(y, my)
    if a.min() < 0 or c.min() < 0:
        return np.inf
    g = float(mx @ my)
    uab, uba = max((x @ my).max(), 0.0), max((y @ mx).max(), 0.0)
    w = uab - min(a.min() * g, a.max() * g)
    return a.max() * uba + max(c.min() * w, c.max() * w) + ra * rc


def _groups(kind, r):
    d, n = 24, 40
    if kind == "clusters":
        cx, cy = r.normal(size=d), r.normal(size=d)
        return cx + 0.4 * r.normal(size=(n, d)), cy + 0.4 * r.normal(size=(n, d))
    if kind == "same":
        c = r.normal(size=d)
        return c + 0.2 * r.normal(size=(n, d)), c + 0.2 * r.normal(size=(n, d))
    if kind == "mixed":
        c = r.normal(size=(3, d))
        return c[r.integers(0, 2, n)] + 0.1 * r.normal(size=(n, d)), c[r.integers(1, 3, n)] + 0.1 * r.normal(size=(n, d))
    if kind == "flat":
        return r.normal(size=(n, d)), r.normal(size=(n, d))
    if kind == "zeros":
        x = r.normal(size=d) + 0.3 * r.normal(size=(n, d))
        x[::7] = 0.0
        return x, np.zeros((n, d))
    if kind == "aligned":  # residuals along one direction: the Cauchy-Schwarz term is tight
        c, e = r.normal(size=d), r.normal(size=d)
        return c + np.outer(r.uniform(0, 1, n), e), c - 0.1 * r.normal(size=d) + np.outer(r.uniform(0, 1, n), e)
    return (r.random((n, d)) < 0.3).astype(float), (r.random((n, d)) < 0.1).astype(float)  # bits


@pytest.mark.parametrize("kind", ["clusters", "same", "mixed", "flat", "zeros", "aligned", "bits"])
def test_bound_holds(kind):
    r = np.random.default_rng(sum(kind.encode()))
    for _ in range(50):
        x, y = _groups(kind, r)
        for mx, my in ((x.mean(0), y.mean(0)), (np.round(3 * x.mean(0)), np.round(3 * y.mean(0))),
                       (x.mean(0), r.normal(size=x.shape[1]))):
            top = _bound(x, y, mx, my)
            scale = max((x * x).sum(1).max(), (y * y).sum(1).max(), 1.0)
            assert (x @ y.T).max() <= top + 1e-9 * scale


def test_binary_bound_on_j():
    r = np.random.default_rng(1)
    for _ in range(100):
        x, y = _groups("bits", r)
        i = x @ y.T
        j = i / np.maximum(x.sum(1)[:, None] + y.sum(1)[None, :] - i, 1.0)
        top = _bound(x, y, x.mean(0), y.mean(0))
        size = x.sum(1).min() + y.sum(1).min() - top
        assert size <= 0 or j.max() <= top / size + 1e-12
