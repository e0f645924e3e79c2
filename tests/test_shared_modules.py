"""A regime's kernels in two modules: kernel (a) by launch shape, the others the
same for every shape, so that a batch size that takes another shape compiles
kernel (a) alone, and the strips of the line form are no shape at all."""

import re

import pytest

from pylcm_b200.codegen import LaunchConfig
from pylcm_b200.engine import SolveEngine
from tests import models as M
from tests.test_codegen import NVRTC, nvrtc_compile

SIZES = [(60, 60), (100, 200), (200, 300), (333, 401), (500, 500), (800, 800)]
BATCHES = [1, 2, 4, 8, 16, 32, 64, 128, 256]


def _kernel_names(src):
    return set(re.findall(r'extern "C" __global__ void __launch_bounds__\([^)]*\) (\w+)\(', src))


@pytest.mark.parametrize("precision,most", [("fp64", 9), ("fp32", 11)])
def test_modules_of_many_batch_sizes(precision, most):
    a, rest = set(), set()
    for grid in SIZES:
        model = M.stochastic_model(4, *grid)
        spec = next(s for s in model.regime_specs if s.name == "working")
        for n in BATCHES:
            eng = SolveEngine(model, precision)
            x, y = eng.kernels(spec, eng.targets_at(spec, 0), M.stochastic_params(), n).sources()
            a.add(x)
            rest.add(y)
    # the others: once, or once per search form (their action tables differ)
    assert len(rest) <= 2
    assert len(a) <= most


CASES = {
    "stochastic": (lambda: M.stochastic_model(4, 500, 500), M.stochastic_params),
    "hc": (lambda: M.hc_model(3, 10, 4, 4, 8), lambda: M.hc_params(0, 4)),
    "taste": (lambda: M.ijrs_dcegm_model(), M.ijrs_params),
}


@pytest.mark.skipif(not NVRTC.exists(), reason="NVRTC not installed")
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_both_modules_compile_and_hold_every_kernel(case, precision):
    mk, mp = CASES[case]
    model, params = mk(), mp()
    n = 0
    for cfg in (None, LaunchConfig(block=128, lanes=4, chunk=256, sb=2)):
        eng = SolveEngine(model, precision, configs=None if cfg is None else {s.name: cfg for s in model.regime_specs})
        for s in eng.specs:
            if s.solver is not None and hasattr(s.solver, "savings_grid"):
                continue
            rk = eng.kernels(s, eng.targets_at(s, min(s.active_periods)), params, 3)
            a, rest = rk.sources()
            assert _kernel_names(a) == {rk.bellman_name()}
            assert _kernel_names(a) | _kernel_names(rest) == _kernel_names(rk.source())
            assert rk.tag not in rest and {rk.atab_name(), rk.sim_name()} <= _kernel_names(rest)
            for src in (a, rest):
                rc, log = nvrtc_compile(src)
                assert rc == 0, log[:2000]
            n += 1
    assert n
