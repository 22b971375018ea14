"""Tile lists at the limits of their arrays, made small: groups of several tiles (as above 2^20 rows),
fewer segments than the order has cuts, and binary rows with more strays than their room holds.
Against the full scan (row slices) bit for bit."""
import numpy as np
import pytest

from evoc import _lib
from test_lists_taken_gpu import bit_clusters, clusters, same_as_slices

pytestmark = pytest.mark.gpu

N = 40000


def _rows(kind, seed):
    if kind == "bits":
        return bit_clusters(N + seed, 32, seed), {"form": _lib.FORM_EXACT_INT}
    x = clusters(N + seed, 96, seed)
    if kind == "i8":
        return np.clip(np.round(127 * x), -127, 127).astype(np.int8), {"form": _lib.FORM_EXACT_INT}
    return x, {"form": _lib.FORM_BF16_RERANK, "certify": 0}


@pytest.mark.parametrize("kind", ["f32", "i8", "bits"])
@pytest.mark.parametrize("limits", ["157,0", "79,0", "20,0", "3,0", "1,0", "157,160", "157,157", "20,23", "5,6"])
def test_groups_and_segments(monkeypatch, kind, limits):
    monkeypatch.setenv("EVOC_LIST_LIMITS", limits)
    x, opts = _rows(kind, int(limits.split(",")[0]))
    same_as_slices(x, 15, **opts)


@pytest.mark.parametrize("nbytes", [33, 128])
def test_more_strays_than_room(nbytes):
    """Half of the rows like one of 20 prototypes, at the pivots' places too, and half like nothing: the
    room for the strays' expanded rows, that of the packed rows, holds an eighth of all rows (33 bytes,
    padded to 64: a sixth)."""
    r = np.random.default_rng(nbytes)
    bits = nbytes * 8
    protos = r.random((20, bits)) < 0.3
    rows = protos[r.integers(0, 20, N)] ^ (r.random((N, bits)) < 0.01)
    odd = np.nonzero(np.arange(N) * 78 // N == (np.arange(N) - 1) * 78 // N)[0]  # 78 pivots: not their rows
    odd = r.permutation(odd)[: 2 * N // 5]
    rows[odd] = r.random((len(odd), bits)) < 0.02
    same_as_slices(np.packbits(rows, axis=1), 15, form=_lib.FORM_EXACT_INT)
