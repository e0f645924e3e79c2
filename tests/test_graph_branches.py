"""The branches of a captured solve: every launch comes after all launches of
the period before and, within a step, kernel (a) after its expectations,
statistics and action table; and the captured solve gives what the launches in
a row give, bit for bit."""

import types

import numpy as np
import pytest

from pylcm_b200 import engine as E
from pylcm_b200 import examples as X
from tests import models as M


class _Stream:
    """A stream that knows, per launch, the set of launches that precede it."""

    def __init__(self):
        self.before = frozenset()
        self.cuda_stream = self

    def record_event(self):
        return self.before

    def wait_event(self, ev):
        self.before |= ev


STEPS = {
    "plain": {"a": ["expect", "expect", "atab", "bellman"], "b": ["expect", "expect", "atab", "bellman"],
              "c": ["atab", "bellman"]},
    "search32": {"a": ["expect", "expect_tc", "stats", "expect", "expect_tc", "atab", "bellman", "egm"],
                 "b": ["expect", "expect_tc", "atab", "bellman"]},
    "egm": {"a": ["egm", "fues", "egm", "egm"], "b": ["egm", "env", "egm", "egm"], "c": ["expect", "atab", "bellman"]},
    "many": {c: ["expect"] * 4 + ["stats", "atab", "bellman"] for c in "abcdefgh"},
    "one": {"a": ["atab", "bellman"]},
}


@pytest.mark.parametrize("case", sorted(STEPS))
def test_order_of_the_branches(case):
    steps = STEPS[case]
    launches = [types.SimpleNamespace(period=p, regime=r, kind=k) for p in (3, 2, 1) for r in steps for k in steps[r]]
    seen = {}

    def op(i):
        def launch(stream):
            seen[i] = stream.before
            stream.before |= {i}
        return launch

    plan = types.SimpleNamespace(
        eng=types.SimpleNamespace(specs=[types.SimpleNamespace(name=r) for r in steps]),
        launches=launches, MAX_LANES=E.SolvePlan.MAX_LANES, _prepared=[op(i) for i in range(len(launches))])
    lanes = E.SolvePlan._lanes(plan)
    assert min(lanes) == 0 and max(lanes) < E.SolvePlan.MAX_LANES
    streams = [_Stream() for _ in range(max(lanes) + 1)]
    E.SolvePlan._run_branches(plan, lanes, streams)
    assert sorted(seen) == list(range(len(launches)))
    assert streams[0].before == frozenset(seen)  # everything joins the capturing stream
    for i, l in enumerate(launches):
        for j in range(i):
            m = launches[j]
            same = m.period == l.period and m.regime == l.regime
            need = m.period != l.period
            need |= same and l.kind not in ("expect", "expect_tc", "stats", "atab")
            need |= l.kind == "stats" and j == i - 1
            need |= l.kind == m.kind == "expect_tc"
            assert not need or j in seen[i], (i, j, l, m)


GRAPHS = {
    "stochastic": (lambda: M.stochastic_model(5, 60, 80), lambda: [M.stochastic_params(beta=b) for b in (0.9, 0.95)]),
    "hc": (lambda: X.hc_model(4, 60, 5, 9, 40), lambda: [X.hc_params(k, 9) for k in range(3)]),
    "dcegm": (M.ijrs_dcegm_model, lambda: [M.ijrs_params(), M.ijrs_params(0.3)]),
    "value_children": (lambda: M.value_children_model(False, 40, 50), lambda: [M.value_children_params()]),
}


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("case", sorted(GRAPHS))
def test_captured_solve_equals_the_launches_in_a_row(case, precision):
    import torch

    model, params = GRAPHS[case][0](), GRAPHS[case][1]()
    a, b = (E.SolveEngine(model, precision).plan(params) for _ in range(2))
    a.run()
    b.capture()
    for t in [*b.V.values(), *b.pol.values()]:
        t.zero_()
    for _ in range(3):
        b.run_graph()
    torch.cuda.synchronize()
    for s in a.V:
        if a.slot[s]:
            np.testing.assert_array_equal(a.V[s].cpu().numpy(), b.V[s].cpu().numpy())
            np.testing.assert_array_equal(a.pol[s].cpu().numpy(), b.pol[s].cpu().numpy())
