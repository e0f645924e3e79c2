"""Grids beyond the line form's limits (its shared memory, its action table, two
groups of actions) keep the search and the launch shape that a regime without
the form gets, in a plain solve and in the server's shape; the grids just
inside take the form.  Results there equal the full search's."""

import dataclasses

import numpy as np
import pytest

from pylcm_b200.engine import SolveEngine, default_config
from pylcm_b200.serving import Server
from tests import models as M

# (wealth, consumption points), in the form?
GRIDS = {
    "2048_actions": ((500, 2048), {"fp32": True, "fp64": True}),
    "2049_actions": ((500, 2049), {"fp32": False, "fp64": False}),
    "3000_actions": ((500, 3000), {"fp32": False, "fp64": False}),
    "long_row": ((9000, 500), {"fp32": False, "fp64": False}),
    "row_of_6000": ((6000, 500), {"fp32": True, "fp64": False}),
    "two_groups": ((500, 16), {"fp32": True, "fp64": True}),
    "below_two_groups": ((500, 15), {"fp32": False, "fp64": False}),
}


def _kernels(model, precision, n, cfg=None):
    spec = next(s for s in model.regime_specs if s.name == "working")
    eng = SolveEngine(model, precision, configs=None if cfg is None else {spec.name: cfg})
    return eng.kernels(spec, eng.targets_at(spec, 0), M.stochastic_params(), n)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_form_by_grid(grid, precision):
    (nw, nc), inside = GRIDS[grid]
    model = M.stochastic_model(3, nw, nc)
    spec = next(s for s in model.regime_specs if s.name == "working")
    plain = _kernels(model, precision, 256)
    served = _kernels(model, precision, 256, Server.SHAPE)
    if inside[precision]:
        assert served._line is not None
        if nc > 16:  # (a batch of fewer pairs takes the full search in double precision)
            assert plain._line is not None
        assert served.smem_bytes if served.source() else 0
    else:
        assert plain._line is None and served._line is None
        assert plain.cfg == default_config(spec, precision, 256)
        assert plain.n_tiles() == -(-spec.n_states // plain.cfg.states_per_tile)
        if precision == "fp32":  # skipping by group statistics where its table fits
            assert plain._groups is not None or nc > plain.GROUP_MAX_CHUNK


@pytest.mark.parametrize("n_consumption", [16, 20, 31, 32])
def test_two_groups_at_every_number_of_threads(n_consumption):
    for n in (1, 2, 4, 8, 20):
        rk = _kernels(M.stochastic_model(3, 100, n_consumption), "fp32", n)
        assert rk._line is None or n_consumption >= 2 * max(rk.LINE_GROUP, rk.line_lanes)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("grid", [(60, 2049), (7000, 40), (9001, 33), (60, 15), (60, 16)])
def test_results_beyond_the_limits(grid, precision):
    import torch

    model, params = M.stochastic_model(3, *grid), [M.stochastic_params()] * 2
    res = []
    for prune in (None, False):
        cfg = None if prune is None else {s.name: dataclasses.replace(default_config(s, precision, 2), prune=False)
                                          for s in model.regime_specs}
        plan = SolveEngine(model, precision, configs=cfg).plan(params)
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
