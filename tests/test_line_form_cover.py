"""The two-axis line form in double precision where the collapsed coordinate and
the law as written round apart: a grid far from zero, so that the law's sum is
off by thousandths of a node.  Which actions are left out may not depend on
that: values within 1e-12 of the full search's, equal policies.

And where the collapsed coordinate falls on a node beside infeasible states
(values of -inf): a weight that one form rounds to zero may not hide or bring
in such a value."""

import dataclasses

import numpy as np
import pytest

from pylcm_b200 import examples as E
from pylcm_b200.engine import SolveEngine, default_config

pytestmark = pytest.mark.gpu


def _next_far(human_capital, hours):
    return human_capital + hours


def _both(model, params, lanes=2, values=None):
    """V and policy of the first regime's last search in the line form and in
    the full search, from the same next-period values."""
    import torch

    out = []
    for prune in (True, False):
        cfg = {s.name: dataclasses.replace(default_config(s, "fp64"), lanes=lanes, sb=1, prune=prune)
               for s in model.regime_specs}
        eng = SolveEngine(model, "fp64", configs=cfg)
        spec = next(s for s in model.regime_specs if s.name == "alive")
        assert (eng.kernels(spec, eng.targets_at(spec, 0), params)._line is not None) == prune
        plan = eng.plan([params])
        plan.run()
        torch.cuda.synchronize()
        if values is not None:
            slot = plan.slot["alive"][1]
            plan.V["alive"][0, slot].copy_(torch.from_numpy(values.reshape(-1)))
            for l, launch in zip(plan.launches, plan._prepare()):
                if l.period == 0:
                    launch(torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
        slot = plan.slot["alive"][0]
        out.append((plan.V["alive"][0, slot].cpu().numpy(), plan.pol["alive"][0, slot].cpu().numpy()))
    return out


def _compare(a, b):
    (va, pa), (vb, pb) = a, b
    np.testing.assert_array_equal(np.isnan(va), np.isnan(vb))
    np.testing.assert_array_equal(np.isfinite(va), np.isfinite(vb))
    fin = np.isfinite(vb)
    assert (np.abs(va - vb)[fin] <= 1e-12 * np.maximum(1.0, np.abs(vb[fin]))).all()
    np.testing.assert_array_equal(pa, pb)


@pytest.fixture
def far_model(monkeypatch):
    real = E.LinSpacedGrid

    def grid(start, stop, n_points):
        if (start, stop) == (1, 5):  # the human-capital axis: steps of 0.37 far from zero
            return real(start=1e11, stop=1e11 + 0.37 * (n_points - 1), n_points=n_points)
        if (start, stop) == (0, 1):  # hours: the law's sums round up by some 0.45 ulp
            stop = 0.70000534
        return real(start=start, stop=stop, n_points=n_points)

    monkeypatch.setattr(E, "LinSpacedGrid", grid)
    monkeypatch.setattr(E, "_hc_next_hc", _next_far)
    monkeypatch.setattr(E, "_hc_next_wealth",
                        lambda wealth, consumption, hours, interest_rate: (1 + interest_rate) * (wealth - consumption) + 20.0 * hours)
    return E.hc_model(3, 257, 12, 2, 130)


@pytest.mark.parametrize("lanes", [2, 8])
def test_coordinates_that_round_apart(far_model, lanes):
    # interior optima with close runners-up, steep along the collapsed axis
    V = np.tile(-30.0 / (np.linspace(0.0, 1000.0, 257) + 2.0)[:, None] + 40.0 * np.arange(12), (2, 1, 1))
    _compare(*_both(far_model, E.hc_params(1, 2, crra=2.0, beta=0.95), lanes, V))


@pytest.mark.parametrize("lanes", [2, 8])
def test_nodes_beside_infeasible_states(monkeypatch, lanes):
    monkeypatch.setattr(E, "_hc_next_hc", lambda human_capital, hours: human_capital + 0.1 * hours)
    model = E.hc_model(3, 130, 41, 2, 64)  # steps of 0.1: the law lands on nodes, one ulp to either side
    rng = np.random.default_rng(1)
    V = np.cumsum(rng.random((2, 130, 41)), axis=1)
    V[:, :, ::3] = -np.inf
    V[:, ::7, 1] = np.nan
    _compare(*_both(model, E.hc_params(1, 2, crra=2.0, beta=0.95), lanes, V))
