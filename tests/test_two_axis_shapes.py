"""Regimes with two continuous states keep the search by collapsed rows where
nobody asks for another: in the server's shape and among the tuner's shapes, as
in a plain solve.  With one continuous state the line form is taken there."""

import dataclasses

import pytest

from pylcm_b200 import autotune
from pylcm_b200.engine import SolveEngine
from pylcm_b200.serving import Server
from tests import models as M

MODELS = {
    "two_axes": (lambda: M.hc_model(4, 1000, 50, 32, 300), lambda: M.hc_params(0, 32), "alive"),
    "one_axis": (lambda: M.stochastic_model(4, 500, 500), M.stochastic_params, "working"),
}


def _kernels(model, params, precision, regime, cfg, n):
    spec = next(s for s in model.regime_specs if s.name == regime)
    eng = SolveEngine(model, precision, configs=None if cfg is None else {regime: cfg})
    return eng.kernels(spec, eng.targets_at(spec, 0), params, n)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", sorted(MODELS))
def test_the_servers_shape(case, precision):
    mk, par, regime = MODELS[case]
    rk = _kernels(mk(), par(), precision, regime, Server.SHAPE, 8)
    assert (rk._line is not None) == (case == "one_axis")


@pytest.mark.parametrize("n", [1, 64])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", sorted(MODELS))
def test_the_tuners_shapes(case, precision, n):
    mk, par, regime = MODELS[case]
    model, params = mk(), par()
    spec = next(s for s in model.regime_specs if s.name == regime)
    plain = _kernels(model, params, precision, regime, None, n)
    cands = autotune.regime_candidates(SolveEngine(model, precision), spec, params, n)
    assert cands[0] == plain.cfg and len(set(cands)) == len(cands) >= 8
    for cfg in cands[:1] + cands[-2:]:
        rk = _kernels(model, params, precision, regime, cfg, n)
        assert (rk._line is None) == (plain._line is None)


def test_tuned_shapes_come_back_from_the_file(monkeypatch, tmp_path):
    import torch

    model, params = M.hc_model(4, 40, 6, 4, 60), M.hc_params(0, 4)
    monkeypatch.setattr(autotune, "CACHE", tmp_path / "autotune.json")
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "no device")
    seen = []
    monkeypatch.setattr(autotune, "_time_regime", lambda m, p, ps, spec, cfg: seen.append(cfg) or float(len(seen)))
    first = autotune.tune(model, "fp32", [params], regimes=["alive"])
    assert seen and not any(c.prune for c in seen)
    timed = len(seen)
    assert autotune.tune(model, "fp32", [params], regimes=["alive"]) == first and len(seen) == timed
    assert all(dataclasses.replace(c) == c and not c.prune for c in first.values())
