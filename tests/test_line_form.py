"""The line form of kernel (a): the exact search that skips action groups on
bounds from expectation rows in shared memory, in both precisions.

CPU: which regimes take it, how its tiles cover a line, the launch shape by
batch size.  GPU: V and policies of the line form against the full search of
the same kernels at line lengths around a strip and a tile, action grids around
a group, several threads per state, one- and two-axis targets.  Both searches
evaluate the surviving actions with the same double arithmetic (in single
precision: re-evaluate the same two candidates), an ulp per operation apart at
most where the compiler fuses differently: V within 1e-12, policies equal
wherever V's runner-up is further than that, i.e. on >= 99.99 % of states."""

import dataclasses

import numpy as np
import pytest

from pylcm_b200.engine import SolveEngine, default_config
from tests import models as M


def _rk(model, params, precision, regime, n_items=1, **cfg):
    spec = next(s for s in model.regime_specs if s.name == regime)
    conf = {spec.name: dataclasses.replace(default_config(spec, precision, n_items), **cfg)} if cfg else None
    eng = SolveEngine(model, precision, configs=conf)
    return eng.kernels(spec, eng.targets_at(spec, 0), params, n_items)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_eligibility(precision):
    rk = _rk(M.stochastic_model(4, 30, 40), M.stochastic_params(), precision, "working", lanes=2)
    assert rk._line is not None and rk._line["line"] == "wealth" and rk._line["scan"] == "consumption"
    rk = _rk(M.hc_model(3, 10, 4, 4, 8), M.hc_params(0, 4), precision, "alive", lanes=2)
    assert rk._line["line"] == "wealth" and rk._line["targets"][0]["coll"]["ob"] == "hours"
    for kw in ({"prune": False}, {"prune_multi": True}, {"collapse": False}):
        assert _rk(M.hc_model(3, 10, 4, 4, 8), M.hc_params(0, 4), precision, "alive", **kw)._line is None
    # a stochastic regime transition: every action reads several targets
    m = M.mass_model()
    assert all(_rk(m, M.mass_params(), precision, s.name, lanes=2)._line is None for s in m.regime_specs if not s.terminal)


@pytest.mark.parametrize("n_wealth", [2, 127, 128, 129, 500])
@pytest.mark.parametrize("lanes,sb", [(1, 1), (2, 4), (8, 2)])
def test_tiles_cover_every_state_once(n_wealth, lanes, sb):
    rk = _rk(M.stochastic_model(3, n_wealth, 40), M.stochastic_params(), "fp32", "working", lanes=lanes, sb=sb)
    per_strip = rk.cfg.block // rk.line_lanes
    parts = -(-n_wealth // rk.line_tile)
    assert rk.n_tiles() == 7 * parts
    seen = np.zeros(7 * n_wealth, dtype=int)
    for tile in range(rk.n_tiles()):  # the kernel's index arithmetic
        line, part = divmod(tile, parts)
        for strip in range(sb):
            pos0 = part * rk.line_tile + strip * per_strip
            if pos0 >= n_wealth:
                break
            pos = np.arange(pos0, min(pos0 + per_strip, n_wealth))
            seen[line * n_wealth + pos] += 1
    assert (seen == 1).all()


def test_launch_shape_by_batch_size():
    shape = lambda n, p: _rk(M.stochastic_model(3, 500, 500), M.stochastic_params(), p, "working", n).cfg  # noqa: E731
    assert not shape(1, "fp64").prune and shape(1, "fp32").prune  # a single double solve: the full search
    assert [shape(n, "fp64").lanes for n in (6, 12, 20, 256)] == [8, 4, 2, 2]
    assert shape(20, "fp64").sb == 1 and shape(40, "fp64").sb == 2


CASES = {
    # (wealth, consumption points): around a strip of 256 / LANES states, around a group of 8
    "edge_strip": (M.stochastic_model, (3, 257, 64), M.stochastic_params),
    "short_line": (M.stochastic_model, (3, 5, 31), M.stochastic_params),
    "few_actions": (M.stochastic_model, (3, 70, 17), M.stochastic_params),
    "below_two_groups": (M.stochastic_model, (3, 70, 15), M.stochastic_params),
    "long_action_grid": (M.stochastic_model, (3, 40, 1500), M.stochastic_params),
    "coarse_actions": (M.stochastic_model, (3, 900, 33), M.stochastic_params),
    "deterministic": (M.retirement_model, (4, 130, 90), M.retirement_params),
    "two_axes": (M.hc_model, (4, 261, 7, 3, 70), lambda: M.hc_params(1, 3)),
    "two_axes_short": (M.hc_model, (4, 33, 5, 4, 16), lambda: M.hc_params(2, 4)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("lanes,sb", [(2, 2), (8, 1), (32, 1)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_line_form_equals_the_full_search(case, lanes, sb, precision):
    import torch

    mk, args, par = CASES[case]
    model, params = mk(*args), [par()] * 2
    res = []
    for prune in (True, False):
        cfg = {s.name: dataclasses.replace(default_config(s, precision, 2), lanes=lanes, sb=sb if prune else 1, prune=prune)
               for s in model.regime_specs}
        plan = SolveEngine(model, precision, configs=cfg).plan(params)
        plan.run()
        torch.cuda.synchronize()
        res.append(plan)
    a, b = res
    for r in a.V:
        va, vb = a.V[r].cpu().numpy(), b.V[r].cpu().numpy()
        np.testing.assert_array_equal(np.isnan(va), np.isnan(vb))
        fin = np.isfinite(vb)
        np.testing.assert_array_equal(np.isfinite(va), fin)
        same = (a.pol[r] == b.pol[r]).cpu().numpy()
        assert same.mean() >= 0.9999, (r, same.mean())
        d = np.abs(va - vb)[fin] / np.maximum(1.0, np.abs(vb[fin]))
        assert d.max(initial=0.0) <= (1e-12 if same.all() or precision == "fp64" else 1e-6), (r, d.max())


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("shape", [(1000, 50, 32, 300), (136, 26, 7, 226)])
def test_two_axes_take_the_full_search_unless_asked(precision, shape):
    nw, nh, ns, nc = shape
    assert _rk(M.hc_model(3, nw, nh, ns, nc), M.hc_params(0, ns), precision, "alive", 3)._line is None
    assert _rk(M.hc_model(3, nw, nh, ns, nc), M.hc_params(0, ns), precision, "alive", 3, lanes=2)._line is not None
