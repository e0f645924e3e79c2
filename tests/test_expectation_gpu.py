"""Kernel (b) against the node-by-node sum in NumPy float64, bit for bit (the
same products, added in node order, divided by the same weight sum), at node
counts around its chunks (8, 16) and row blocks (16), with weights of zero and
values that are not finite; the tensor-core table within 2e-6 of it."""

import numpy as np
import pytest

from pylcm_b200 import examples as E
from pylcm_b200.engine import SolveEngine

pytestmark = pytest.mark.gpu


def _sum(W, V):
    acc = np.zeros((W.shape[0], V.shape[1]))
    sw = np.zeros(W.shape[0])
    with np.errstate(invalid="ignore"):
        for j in range(W.shape[1]):
            w = W[:, j, None]
            acc = acc + np.where((w == 0.0) & ~np.isfinite(V[j]), 0.0, w * V[j])
            sw = sw + W[:, j]
        return acc / np.where(sw > 0.0, sw, 1.0)[:, None]


@pytest.mark.parametrize("n", [2, 7, 8, 15, 16, 17, 24, 31, 33, 64])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_expectation_is_the_node_sum(n, precision):
    import torch

    rng = np.random.default_rng(n)
    model = E.hc_model(3, 43, 3, n, 20)
    params = E.hc_params(1, n)
    P = params["shock_transition"]
    P[rng.random((n, n)) < 0.4] = 0.0  # rows no longer sum to one
    P[n // 2] = 0.0
    plan = SolveEngine(model, precision).plan([params])
    plan.run()
    V = plan.V["alive"][0, plan.slot["alive"][1]].cpu().numpy().reshape(n, -1)
    V = np.where(np.isfinite(V), V, -3.0) + rng.normal(size=V.shape)
    cols = rng.permutation(V.shape[1])
    V[:, cols[0]] = -np.inf
    V[rng.random(n) < 0.5, cols[1]] = -np.inf
    V[0, cols[2]], V[n - 1, cols[2]] = -np.inf, np.inf
    V[n // 2, cols[3]], V[0, cols[4]] = np.nan, np.inf
    V[rng.random(n) < 0.5, cols[5]] = np.nan
    V[0, cols[5]] = -np.inf
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
    if e32 is not None:
        got = e32[0].cpu().numpy().astype(np.float64)
        fin = np.isfinite(V).all(axis=0)
        assert (np.abs(got - want)[:, fin] <= 2e-6 * np.maximum(1.0, np.abs(want[:, fin]))).all()
        np.testing.assert_array_equal(got[:, ~fin], want[:, ~fin].astype(np.float32))
