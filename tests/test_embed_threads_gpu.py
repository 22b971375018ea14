"""Node embeddings of several widths at once, a thread and a context each: the launches of one must not
depend on what another asks of the same kernel.  Every result equals the one made alone."""
import threading

import numpy as np
import pytest

import evoc
from evoc import _lib
from oracle import label_prop as L
from test_label_prop_gpu import _tuple

pytestmark = pytest.mark.gpu


def test_widths_at_once(monkeypatch):
    n, widths, runs = 400, [2, 8, 3, 8, 2, 7, 4, 8], 12
    rng = np.random.default_rng(3)
    d = rng.integers(1, 12, n)
    indptr = np.concatenate([[0], np.cumsum(d)]).astype(np.int64)
    m = int(indptr[-1])
    g = _tuple(L.Csr(indptr, rng.integers(0, n, m).astype(np.int32), (0.05 + 0.95 * rng.random(m)).astype(np.float32),
                     (n, n)))
    alone = {w: evoc.node_embedding(g, w, 60, None, 0.1, 1.0, 0.5, np.random.RandomState(w)) for w in set(widths)}
    mine = threading.local()

    def context(device=0):
        if not hasattr(mine, "ctx"):
            mine.ctx = _lib.Context(device)
        return mine.ctx

    monkeypatch.setattr(_lib, "context", context)
    wrong = []

    def work(w):
        try:
            for _ in range(runs):
                emb = evoc.node_embedding(g, w, 60, None, 0.1, 1.0, 0.5, np.random.RandomState(w))
                if not np.array_equal(emb.view(np.uint32), alone[w].view(np.uint32)):
                    wrong.append((w, "differs"))
        except Exception as e:
            wrong.append((w, repr(e)))

    threads = [threading.Thread(target=work, args=(w,)) for w in widths]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
