"""The launches a context reports for the small form: a product and a selection for each stretch of rows
whose scores stay within 64 MB."""
import numpy as np
import pytest

import evoc
from evoc import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,stretches", [(300, 1), (4000, 1), (4300, 2), (5000, 2)])
def test_small_form(n, stretches):
    x = np.random.default_rng(n).integers(-127, 128, size=(n, 48)).astype(np.int8)
    rows = (64 << 20) // ((n + 255) // 256 * 256 * 4) // 128 * 128
    assert stretches == -(-n // rows)
    evoc.knn_graph(x, evoc.KnnGraphOptions(n_neighbors=30, form="exact_int"))
    assert _lib.context(0).launches() == 2 * stretches  # host rows are copied, not launched
