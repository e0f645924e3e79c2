"""The line form where the next period's values are -inf, NaN or +inf: one
search, both forms on the same values, one and two axes, both precisions.  The
bounds of a group of actions and the evaluation without branches have rules of
their own for such values.  NaN and infinite results in the same places; values
within 1e-12 wherever the policies agree (the same arithmetic), and they agree
but for float near-ties of the single-precision search."""

import dataclasses

import numpy as np
import pytest

from pylcm_b200.engine import SolveEngine, default_config
from tests import models as M

pytestmark = pytest.mark.gpu

MODELS = {
    "one_axis": (lambda: M.stochastic_model(3, 260, 130), M.stochastic_params, "working", (7, 260)),
    "two_axes": (lambda: M.hc_model(3, 133, 9, 4, 70), lambda: M.hc_params(1, 4), "alive", (4, 133, 9)),
}


def _values(kind, shape, rng):
    V = np.cumsum(rng.random(shape), axis=1) ** 0.7 - 5.0
    if kind == "low_infeasible":  # no state below a wealth is feasible
        V[:, : shape[1] // 4] = -np.inf
    elif kind == "scattered":
        V[rng.random(shape) < 0.02] = -np.inf
        V[rng.random(shape) < 0.005] = np.nan
    elif kind == "nan_top":  # as it spreads from beyond the grid
        V[:, -shape[1] // 3:] = np.nan
    elif kind == "nan_row":
        V[1] = np.nan
        V[2] = -np.inf
    elif kind == "plus_inf":
        V[rng.random(shape) < 0.01] = np.inf
        V[0, shape[1] // 2] = -np.inf
    return V


@pytest.mark.parametrize("kind", ["low_infeasible", "scattered", "nan_top", "nan_row", "plus_inf"])
@pytest.mark.parametrize("lanes", [2, 8])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", sorted(MODELS))
def test_forms_agree_beside_values_that_are_not_finite(case, precision, lanes, kind):
    import torch

    mk, par, regime, shape = MODELS[case]
    model, params = mk(), par()
    V1 = _values(kind, shape, np.random.default_rng(len(kind)))
    out = []
    for prune in (True, False):
        cfg = {s.name: dataclasses.replace(default_config(s, precision), lanes=lanes, sb=1, prune=prune)
               for s in model.regime_specs}
        plan = SolveEngine(model, precision, configs=cfg).plan([params])
        plan.run()
        for name, V in plan.V.items():  # every regime's next values, whichever is read
            k = plan.slot[name].get(1)
            if k is not None and V[0, k].numel() == V1.size:
                V[0, k].copy_(torch.from_numpy(V1.reshape(-1)))
        for l, launch in zip(plan.launches, plan._prepare()):
            if l.period == 0:
                launch(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        plan.check_status()
        k = plan.slot[regime][0]
        out.append((plan.V[regime][0, k].cpu().numpy(), plan.pol[regime][0, k].cpu().numpy()))
    (va, pa), (vb, pb) = out
    np.testing.assert_array_equal(np.isnan(va), np.isnan(vb))
    np.testing.assert_array_equal(va[np.isinf(vb)], vb[np.isinf(vb)])
    np.testing.assert_array_equal(np.isinf(va), np.isinf(vb))
    same = pa == pb
    assert same.mean() >= (1.0 if precision == "fp64" else 0.999), same.mean()
    fin = np.isfinite(vb)
    with np.errstate(invalid="ignore"):
        d = np.abs(va - vb) / np.maximum(1.0, np.abs(vb))
    assert d[fin & same].max(initial=0.0) <= 1e-12
    assert d[fin].max(initial=0.0) <= 1e-6
