"""Branches of a captured solve are paid for once per solver, when the graph is
instantiated (23 ms for the 40-period single-precision benchmark at 5 branches,
87 at 8): the number of streams that a period forks to and joins is bounded."""

import types

import pytest

from pylcm_b200 import engine as E
from tests.test_graph_branches import STEPS, _Stream


@pytest.mark.parametrize("case", sorted(STEPS))
def test_waits_of_a_period(case):
    waits = 0

    class Stream(_Stream):
        def wait_event(self, ev):
            nonlocal waits
            waits += 1
            super().wait_event(ev)

    steps = STEPS[case]
    launches = [types.SimpleNamespace(period=p, regime=r, kind=k) for p in (2, 1) for r in steps for k in steps[r]]
    plan = types.SimpleNamespace(
        eng=types.SimpleNamespace(specs=[types.SimpleNamespace(name=r) for r in steps]), launches=launches,
        MAX_LANES=E.SolvePlan.MAX_LANES, _prepared=[lambda stream: None] * len(launches))
    lanes = E.SolvePlan._lanes(plan)
    E.SolvePlan._run_branches(plan, lanes, [Stream() for _ in range(max(lanes) + 1)])
    # fork and join of four branches, and every step's own waits
    assert waits / 2 <= 8 + 4 * len(steps)
    assert max(lanes) <= 4
