"""The search form and launch shape of a batch: lines that fill no CTA and short
action grids keep the full search or take several threads per state, long ones
the line form; every shape that the rule can choose gives the full search's
values and policies."""

import dataclasses

import numpy as np
import pytest

from pylcm_b200.engine import SolveEngine, default_config
from tests import models as M


def _kernels(wealth, consumption, n, precision):
    model = M.stochastic_model(3, wealth, consumption)
    spec = next(s for s in model.regime_specs if s.name == "working")
    eng = SolveEngine(model, precision)
    return eng.kernels(spec, eng.targets_at(spec, 0), M.stochastic_params(), n)


# (wealth, consumption, instances): measured at least a quarter slower in the line form at any number of threads
FULL = [(24, 60, 400), (40, 105, 340), (62, 60, 384), (62, 105, 219), (100, 60, 238), (128, 105, 106), (200, 60, 119),
        (300, 60, 397), (800, 30, 298), (800, 60, 149)]
# and at least a quarter faster
LINE = [(62, 400, 288), (100, 800, 89), (128, 400, 140), (200, 400, 89), (300, 400, 60), (500, 250, 57), (500, 500, 256),
        (800, 400, 22)]


@pytest.mark.parametrize("case", FULL)
def test_full_search_in_double_precision(case):
    rk = _kernels(*case, "fp64")
    assert rk._line is None and rk.cfg == dataclasses.replace(default_config(rk.spec, "fp64", case[2]), prune=False)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", LINE)
def test_line_form(case, precision):
    rk = _kernels(*case, precision)
    assert rk._line is not None
    # a CTA's threads are at least a third used
    assert case[0] * rk.line_lanes >= 85


@pytest.mark.parametrize("case", [(24, 30, 496), (40, 30, 298), (62, 30, 192)])
def test_short_lines_and_few_actions_in_single_precision(case):
    assert _kernels(*case, "fp32")._line is None


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", [(62, 400, 60), (24, 801, 120), (33, 60, 9), (257, 131, 40)])
def test_chosen_shape_equals_the_full_search(case, precision):
    import torch

    wealth, consumption, n = case
    model = M.stochastic_model(3, wealth, consumption)
    params = [M.stochastic_params(crra=1.5 + 0.5 * (k % 5)) for k in range(n)]
    res = []
    for full in (False, True):
        cfg = {s.name: dataclasses.replace(default_config(s, precision, n), prune=False) for s in model.regime_specs}
        plan = SolveEngine(model, precision, configs=cfg if full else None).plan(params)
        plan.run()
        torch.cuda.synchronize()
        plan.check_status()
        res.append(plan)
    a, b = res
    for r in a.V:
        va, vb = a.V[r].cpu().numpy(), b.V[r].cpu().numpy()
        np.testing.assert_array_equal(np.isfinite(va), np.isfinite(vb))
        same = (a.pol[r] == b.pol[r]).cpu().numpy()
        assert same.mean() >= 0.9999
        fin = np.isfinite(vb)
        d = np.abs(va - vb)[fin] / np.maximum(1.0, np.abs(vb[fin]))
        assert d[same[fin]].max(initial=0.0) <= 1e-12
        assert d.max(initial=0.0) <= (1e-12 if precision == "fp64" else 1e-6)
