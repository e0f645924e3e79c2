"""Action grids that descend (a logarithmic grid from its largest point down):
the actions that meet a budget constraint are then no prefix of the grid, so
neither the search nor the simulation may stop at one."""

import dataclasses

import numpy as np
import pytest

from oracle.grid_search import solve as oracle_solve
from oracle.simulate import simulate as oracle_simulate
from pylcm_b200 import LinSpacedGrid, LogSpacedGrid
from pylcm_b200 import examples as E
from pylcm_b200.engine import SolveEngine, default_config
from tests.conftest import rel_err

N_WEALTH, N_CONS = 60, 70


@pytest.fixture
def model(monkeypatch):
    def grid(start, stop, n_points):
        if n_points == N_CONS:
            return LogSpacedGrid(start=stop, stop=start, n_points=n_points)
        return LinSpacedGrid(start=start, stop=stop, n_points=n_points)

    monkeypatch.setattr(E, "LinSpacedGrid", grid)
    return E.stochastic_model(4, N_WEALTH, N_CONS)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_no_prefix_of_a_descending_grid(model, precision):
    up = E.retirement_model(4, 30, 40)
    for m, params, prefix in ((model, E.stochastic_params(), False), (up, E.retirement_params(), True)):
        spec = next(s for s in m.regime_specs if s.name == "working")
        eng = SolveEngine(m, precision, configs={spec.name: default_config(spec, precision)})
        rk = eng.kernels(spec, eng.targets_at(spec, 0), params)
        assert (rk._budget_bound() is not None) == prefix
        assert (rk._line["budget"] is not None) == prefix


@pytest.mark.gpu
@pytest.mark.parametrize("prune", [True, False])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_solve_matches_the_oracle(model, precision, prune):
    params = E.stochastic_params()
    cfg = {s.name: dataclasses.replace(default_config(s, precision), prune=prune) for s in model.regime_specs}
    V, _ = SolveEngine(model, precision, configs=cfg).solve(params)
    Vo, _ = oracle_solve(model, params)
    for p in Vo:
        for r in Vo[p]:
            # single precision: the top two of a float search, re-evaluated
            assert rel_err(V[p][r].cpu().numpy(), Vo[p][r]) < (1e-12 if precision == "fp64" else 1e-6), (p, r)


@pytest.mark.gpu
def test_simulation_matches_the_oracle(model):
    params, n = E.stochastic_params(), 75
    rng = np.random.default_rng(2)
    ic = {"wealth": rng.uniform(1, 300, n), "income": rng.normal(0, 0.1, n), "age": np.zeros(n),
          "regime_id": np.zeros(n, dtype=int)}
    res = model.simulate(params=params, initial_conditions=ic, seed=7)
    ora = oracle_simulate(model, params, ic, seed=7)
    for p in ora:
        np.testing.assert_array_equal(res.periods[p]["regime_id"], ora[p]["regime_id"])
        for name in ("wealth", "income"):
            np.testing.assert_allclose(res.periods[p]["states"][name], ora[p]["states"][name], rtol=1e-9, atol=1e-9,
                                       equal_nan=True)
