"""The server's launch shape of a regime that is neither tuned nor given: in
double precision short action grids keep the full search."""

import types

import pytest

from pylcm_b200.engine import SolveEngine
from pylcm_b200.serving import Server
from tests import models as M


@pytest.mark.parametrize("precision,actions,line", [("fp64", 60, False), ("fp64", 255, False), ("fp64", 256, True),
                                                    ("fp64", 500, True), ("fp32", 60, True), ("fp32", 500, True)])
def test_search_form_by_actions(precision, actions, line):
    model = M.stochastic_model(4, 300, actions)
    spec = next(s for s in model.regime_specs if s.name == "working")
    srv = types.SimpleNamespace(precision=precision, SHAPE=Server.SHAPE, LINE_ACTIONS_FP64=Server.LINE_ACTIONS_FP64)
    eng = SolveEngine(model, precision, configs={s.name: Server.shape(srv, s) for s in model.regime_specs})
    rk = eng.kernels(spec, eng.targets_at(spec, 0), M.stochastic_params(), 32)
    assert (rk._line is not None) == line and rk.cfg.block == Server.SHAPE.block
