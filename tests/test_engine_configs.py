"""A launch shape put into, changed in or taken out of `SolveEngine.configs`
holds for the next plan, also of a batch size that was planned before."""

import dataclasses

import pytest

from pylcm_b200.codegen import LaunchConfig
from pylcm_b200.engine import SolveEngine
from tests import models as M


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_changed_shapes_are_taken(precision):
    model, params = M.stochastic_model(4, 30, 40), M.stochastic_params()
    eng = SolveEngine(model, precision)
    spec = next(s for s in model.regime_specs if s.name == "working")
    get = lambda n=3: eng.kernels(spec, eng.targets_at(spec, 0), params, n)  # noqa: E731
    first = get()
    shape = LaunchConfig(block=128, lanes=4, chunk=256, sb=2)
    eng.configs["working"] = shape
    asked = get()
    assert asked.cfg == shape and asked is not first
    eng.configs["working"] = dataclasses.replace(shape, prune=False)
    assert get().cfg == eng.configs["working"] and get()._line is None
    eng.configs["working"] = shape
    assert get() is asked  # kernels made before are kept
    del eng.configs["working"]
    assert get() is first
