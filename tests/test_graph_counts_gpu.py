"""The prefix sums of the fuzzy graph's counts: one launch up to 4,096 of them, three above; results on
both sides of the line against a host merge, and the launches that the context reports."""
import numpy as np
import pytest

import evoc
from evoc import _lib
from test_graph_rows_gpu import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("symmetrize", [True, False])
def test_small_graphs_have_few_launches(symmetrize):
    launches = {}
    for n in (1, 33, 1000, 4095, 4096, 4097):
        r = np.random.default_rng(n)
        ind = np.stack([(np.arange(n) + s) % n for s in (0, 1, 5, 17)], 1).astype(np.int32)
        dst = np.sort(r.random((n, 4)).astype(np.float32), axis=1)
        dst[:, 0] = 0.0
        if n > 17:
            _compare(ind, dst, 4.0, symmetrize)
        evoc.neighbor_graph_csr(4.0, ind, dst, symmetrize)
        launches[n] = _lib.context(0).launches()
    assert len({launches[n] for n in (1, 33, 1000, 4095, 4096)}) == 1
    assert launches[4097] - launches[4096] == (4 if symmetrize else 2)
