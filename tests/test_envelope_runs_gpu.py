"""The envelopes' scans behind run ranges, bit-identical to the oracle (every
step is rounded as the oracle rounds it): row lengths around a run of 16
segments and a CTA, rows ascending already (no sort), shuffled candidates
(every run covers the whole range), dead runs, infinite values and repeated
abscissae."""

import numpy as np
import pytest

from tests.test_envelopes_gpu import _gpu, _oracle, _rows, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ltm", "rfc", "mss"])
@pytest.mark.parametrize("n", [2, 16, 17, 18, 33, 257, 513])
@pytest.mark.parametrize("shape", ["ascending", "folded", "shuffled", "dead_runs", "ties"])
def test_rows_match_the_oracle(kind, n, shape):
    G, P, V, M = _rows(2, n, seed=n)
    rng = np.random.default_rng(n)
    if shape == "ascending":
        o = np.argsort(np.where(np.isnan(G), np.inf, G), axis=1, kind="stable")
        G, P, V, M = (np.take_along_axis(x, o, axis=1) for x in (G, P, V, M))
    elif shape == "shuffled":
        o = np.stack([rng.permutation(n) for _ in range(2)])
        G, P, V, M = (np.take_along_axis(x, o, axis=1) for x in (G, P, V, M))
    elif shape == "dead_runs":
        dead = (np.arange(n) // 16) % 3 == 1
        G, P, V = (np.where(dead, np.nan, x) for x in (G, P, V))
        V = np.where(rng.random(V.shape) < 0.05, -np.inf, V)
        M = np.where(dead, 0.0, M)
    elif shape == "ties":
        G = np.where(np.isnan(G), G, np.round(G, 1))
    n_out = 2 * n + 3
    got = _gpu(kind, G, P, V, M, n_out)
    for r in range(2):
        with np.errstate(all="ignore"):
            _same([x[r] for x in got], _oracle(kind, G[r], P[r], V[r], M[r], n_out))
