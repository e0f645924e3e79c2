"""FUES with a bounded look-ahead on rows whose drops, jumps and next same-segment
candidates lie on either side of the window and of 32 candidates: the rows the
oracle keeps."""

import numpy as np
import pytest

from oracle.fues import refine
from tests.test_fues_gpu import _gpu_fues, _same

pytestmark = pytest.mark.gpu


def _row(kind, n, rng):
    a = np.sort(rng.uniform(0, 10, n))
    i = np.arange(n)
    if kind == "alternating":
        other = i % 2 == 1
    elif kind == "runs":  # runs of 1 to 70 candidates of either branch
        ends = np.cumsum(rng.integers(1, 70, n))
        other = np.searchsorted(ends, i, side="right") % 2 == 1
    else:  # long dominated stretches
        other = rng.random(n) < 0.04
    c = np.where(other, 1.5 + 0.6 * a, 0.5 + 0.3 * a)
    g = a + c
    v = np.log(c) + 0.2 * np.sqrt(a + 1) + np.where(other, 0.7, 0.0) - 0.15 * i / n
    if kind == "dominated":
        v = np.where(other, v, v - 0.3 * rng.random(n))
    gone = rng.random(n) < 0.02
    return np.where(gone, np.nan, g), c, np.where(gone, np.nan, v), a


@pytest.mark.parametrize("window", [1, 2, 10, 31, 32, 33, 64, 500])
@pytest.mark.parametrize("kind", ["alternating", "runs", "dominated"])
def test_bounded_look_ahead(kind, window):
    n, n_out = 333, 700
    rng = np.random.default_rng(window)
    rows = [_row(kind, n, rng) for _ in range(4)]
    G, C, V, S = (np.array(x) for x in zip(*rows))
    go, co, vo, nk = _gpu_fues(G, C, V, S, n_out, window=window)
    for r in range(len(rows)):
        rg, rc, rv, k = refine(G[r], C[r], V[r], S[r], n_out, n_points_to_scan=window)
        assert nk[r] == k
        for got, want in ((go[r], rg), (co[r], rc), (vo[r], rv)):
            _same(got, want)
