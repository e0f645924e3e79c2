"""Subjects per warp of the simulation kernel: the draws and the results of a
subject do not depend on how many subjects its warp takes in turn (bit for
bit: each subject's search and draws are the same operations), at subject
counts around a warp and a tile."""

import numpy as np
import pytest

from pylcm_b200 import simulate as S
from tests import models as M


def test_subjects_per_warp():
    assert [S.subjects_per_warp(n) for n in (1, 10_000, 18_943, 18_944, 160_000, 640_000)] == [1, 1, 1, 2, 16, 32]
    assert S.subjects_per_warp(10**9) == 32


CASES = {
    "stochastic": (lambda: M.stochastic_model(5, 40, 60), M.stochastic_params,
                   lambda rng, n: {"wealth": rng.uniform(1, 60, n), "income": rng.normal(0, 0.25, n)}),
    "human_capital": (lambda: M.hc_model(4, 30, 6, 5, 25), lambda: M.hc_params(1, 5),
                      lambda rng, n: {"wealth": rng.uniform(0, 900, n), "human_capital": rng.uniform(1, 5, n),
                                      "shock": rng.integers(0, 5, n).astype(float)}),
}


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 257])
@pytest.mark.parametrize("case", sorted(CASES))
def test_results_do_not_depend_on_subjects_per_warp(case, n, monkeypatch):
    mk, par, ini = CASES[case]
    model, params = mk(), par()
    rng = np.random.default_rng(n)
    ic = {**ini(rng, n), "regime_id": np.zeros(n, dtype=int)}
    V = model.solve(params=params, log_level="off")
    out = []
    for spw in (1, 4, 32):
        monkeypatch.setattr(S, "subjects_per_warp", lambda total, spw=spw: spw)
        out.append(model.simulate(params=params, initial_conditions=ic, period_to_regime_to_V_arr=V, log_level="off", seed=3))
    for other in out[1:]:
        for p in out[0].periods:
            a, b = out[0].periods[p], other.periods[p]
            np.testing.assert_array_equal(a["regime_id"], b["regime_id"])
            np.testing.assert_array_equal(a["value"], b["value"])
            for group in ("states", "actions"):
                for k in a[group]:
                    np.testing.assert_array_equal(a[group][k], b[group][k])
