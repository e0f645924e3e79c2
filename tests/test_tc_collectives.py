"""The tensor-core expectation's collectives run on converged warps.

CPU: every tensor-memory load waits for its warp's lanes first.  GPU: tables of
several blocks of 16 rows whose columns are finite, -inf, NaN and +inf by turns
within a warp (the lanes take paths of different lengths between two loads)
against the node-by-node sum."""

import re
from pathlib import Path

import numpy as np
import pytest

import pylcm_b200
from pylcm_b200 import examples as E
from pylcm_b200.engine import SolveEngine
from tests.test_expectation_gpu import _sum


def test_loads_wait_for_the_warp():
    src = (Path(pylcm_b200.__file__).parent / "csrc" / "kernels" / "lcm_tc.cuh").read_text()
    src = re.sub(r"//[^\n]*", "", src)
    loads = [m.start() for m in re.finditer(r"tcgen05\.ld\.", src)]
    assert loads
    for at in loads:
        body = src[src.rindex("__device__", 0, at):at]
        assert "__syncwarp();" in body


@pytest.mark.gpu
@pytest.mark.parametrize("n", [17, 48, 64])
def test_lanes_of_different_paths(n):
    import torch

    rng = np.random.default_rng(n)
    model = E.hc_model(3, 67, 3, n, 20)
    params = E.hc_params(1, n)
    P = params["shock_transition"]
    P[rng.random((n, n)) < 0.5] = 0.0
    plan = SolveEngine(model, "fp32").plan([params])
    plan.run()
    V = rng.normal(size=(n, 67 * 3))
    c = np.arange(V.shape[1])
    V[:, c % 5 == 1] = -np.inf
    V[0, c % 5 == 2] = np.nan
    V[n - 1, c % 5 == 3] = np.inf
    V[rng.random(n) < 0.5, 0] = -np.inf
    plan.V["alive"][0, plan.slot["alive"][1]].copy_(torch.from_numpy(V.reshape(-1)))
    stream = torch.cuda.current_stream().cuda_stream
    for l, launch in zip(plan.launches, plan._prepare()):
        if l.period == 0 and l.kind in ("expect", "expect_tc"):
            launch(stream)
    torch.cuda.synchronize()
    plan.check_status()
    want = _sum(P, V)
    (e64, e32), = [(a, b) for (src, tg, t), (a, b, _, _) in plan.ev.items() if t == "alive" and src == "alive"]
    np.testing.assert_array_equal(e64[0].cpu().numpy(), want)
    got = e32[0].cpu().numpy().astype(np.float64)
    fin = np.isfinite(V).all(axis=0)
    np.testing.assert_array_equal(got[:, ~fin], want[:, ~fin].astype(np.float32))
    assert (np.abs(got - want)[:, fin] <= 2e-6 * np.maximum(1.0, np.abs(want[:, fin]))).all()
