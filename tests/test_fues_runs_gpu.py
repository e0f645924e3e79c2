"""The shared-memory FUES kernel where its fast paths begin and end, against
the oracle: rows of 0, 1, 16 and 17 descents (unsorted, merged by ranks, by the
bitonic network), row lengths around a warp, a CTA and its longest row, long
runs of dropped candidates (more than the 32 the warp tests at once), more runs
of plain steps than the CTA keeps for copying, and bounded look-aheads.  Kept
sets identical, values within 1e-12 (crossings may differ by an ulp: fused
multiply-add), as in test_fues_gpu."""

import numpy as np
import pytest

from oracle.fues import refine
from tests.test_fues_gpu import _gpu_fues, _same

pytestmark = pytest.mark.gpu


def _check(G, C, V, S, window=0):
    n_out = 2 * G.shape[1] + 2
    go, co, vo, nk = _gpu_fues(G, C, V, S, n_out, window=window)
    for r in range(G.shape[0]):
        rg, rc, rv, k = refine(G[r], C[r], V[r], S[r], n_out, **({"n_points_to_scan": window} if window else {}))
        assert nk[r] == k
        _same(go[r], rg)
        _same(co[r], rc)
        _same(vo[r], rv)


def _two_branches(rng, n, switch_every=None):
    """Candidates of two concave branches over the same abscissae; which one
    holds a candidate changes in blocks (dropped blocks, jumps at their
    borders)."""
    a = np.sort(rng.uniform(0.0, 10.0, n))
    block = switch_every or max(2, n // 6)
    upper = (np.arange(n) // block) % 2 == 0
    c = np.where(upper, 1.5 + 0.6 * a, 0.5 + 0.3 * a)
    g = np.sort(a + 2.0 * rng.uniform(0.4, 1.0))
    v = np.log(c) + 0.2 * np.sqrt(a + 1) + np.where(upper, 0.8, 0.0)
    return g, c, v, g - c


def _with_descents(rng, row, k):
    """The row's candidates in k + 1 ascending runs."""
    n = len(row[0])
    perm = np.arange(n)
    if k:
        run = rng.integers(0, k + 1, n)
        perm = np.concatenate([np.flatnonzero(run == r) for r in range(k + 1)])
    return [x[perm] for x in row]


@pytest.mark.parametrize("n", [2, 31, 33, 255, 257, 1024, 2049])
@pytest.mark.parametrize("descents", [0, 1, 16, 17, 40])
def test_sorting_paths(n, descents):
    rng = np.random.default_rng(1000 * n + descents)
    rows = [_with_descents(rng, _two_branches(rng, n), min(descents, n - 1)) for _ in range(2)]
    G, C, V, S = (np.stack(x) for x in zip(*rows))
    dead = rng.random(G.shape) < 0.01
    G, V = np.where(dead, np.nan, G), np.where(dead, np.nan, V)
    _check(G, C, V, S)


@pytest.mark.parametrize("block", [1, 2, 5, 31, 70])
@pytest.mark.parametrize("window", [0, 1, 40])
def test_drops_jumps_and_runs(block, window):
    rng = np.random.default_rng(block)
    rows = [_two_branches(rng, 600, block) for _ in range(2)]
    G, C, V, S = (np.stack(x) for x in zip(*rows))
    _check(G, C, V, S, window)


def test_longest_row():
    rng = np.random.default_rng(5)
    G, C, V, S = (np.stack([x]) for x in _with_descents(rng, _two_branches(rng, 4096, 97), 3))
    _check(G, C, V, S)
