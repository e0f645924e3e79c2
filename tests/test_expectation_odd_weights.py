"""Expectations beside weights that are negative or not finite: transition rows
that are no distribution reach the kernels (the checks of the transitions only
warn, and batches and the server do without them).  Such a weight turns a value
of -inf into +inf, or makes the row NaN, so the rule that takes -inf and NaN out
of the sums as bits does not hold for it.

CPU: the tensor-core kernel reads the flag of such weights, which a few threads
set while others own no row, behind a barrier.  GPU: both tables against the
node-by-node sum in NumPy float64, at row counts on the bit path (more than 8
rows) around a block of 16 rows and a warp."""

import re
from pathlib import Path

import numpy as np
import pytest

import pylcm_b200
from pylcm_b200 import examples as E
from pylcm_b200.engine import SolveEngine
from tests.test_expectation_gpu import _sum


def test_the_flag_is_read_behind_a_barrier():
    src = (Path(pylcm_b200.__file__).parent / "csrc" / "kernels" / "lcm_tc.cuh").read_text()
    src = re.sub(r"//[^\n]*", "", src)
    set_at = src.index("Wodd = 1")
    read_at = re.search(r"\|\| Wodd", src).start()
    assert "__syncthreads()" in src[set_at:read_at]


WEIGHTS = {"negative": -0.4, "nan": np.nan, "inf": np.inf, "minus_inf": -np.inf}


@pytest.mark.gpu
@pytest.mark.parametrize("n", [9, 16, 17, 32, 33])
@pytest.mark.parametrize("kind", sorted(WEIGHTS))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_odd_weights_beside_infinite_and_nan_values(n, kind, precision):
    import torch

    rng = np.random.default_rng(n)
    model = E.hc_model(3, 61, 4, n, 20)
    params = [E.hc_params(k, n) for k in range(3)]
    rows = (0, n - 1, n // 2)  # of the first warp, of the last owner of a row, in between
    for k, p in enumerate(params):
        P = p["shock_transition"]
        P[rng.random((n, n)) < 0.2] = 0.0
        if k < 2:  # the third instance's weights are a distribution's
            P[rows[k], 1] = WEIGHTS[kind]
            P[rows[2], n - 2] = WEIGHTS[kind]
    plan = SolveEngine(model, precision).plan(params)
    plan.run()
    slot = plan.slot["alive"][1]
    Vs = []
    for k in range(3):
        V = plan.V["alive"][k, slot].cpu().numpy().reshape(n, -1)
        V = np.where(np.isfinite(V), V, -3.0) + rng.normal(size=V.shape)
        cols = rng.permutation(V.shape[1])
        V[:, cols[0]] = -np.inf
        V[1, cols[1:8]] = -np.inf  # on the odd weights
        V[n - 2, cols[4:12]] = -np.inf
        V[1, cols[8:10]] = np.nan
        V[rng.random(n) < 0.7, cols[10]] = -np.inf
        V[1, cols[11]] = np.inf
        V[:, cols[12]] = -np.inf
        V[0, cols[12]] = np.nan
        plan.V["alive"][k, slot].copy_(torch.from_numpy(V.reshape(-1)))
        Vs.append(V)
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(5):  # (which threads were ahead of the flag was a matter of timing)
        for l, launch in zip(plan.launches, plan._prepare()):
            if l.period == 0 and l.kind in ("expect", "expect_tc"):
                launch(stream)
        torch.cuda.synchronize()
        plan.check_status()
        (e64, e32), = [(a, b) for (src, tg, t), (a, b, _, _) in plan.ev.items() if t == "alive" and src == "alive"]
        for k, V in enumerate(Vs):
            P = params[k]["shock_transition"]
            want = _sum(P, V)
            np.testing.assert_array_equal(e64[k].cpu().numpy(), want)
            if e32 is None:
                continue
            got = e32[k].cpu().numpy().astype(np.float64)
            fin = np.isfinite(V).all(axis=0)
            np.testing.assert_array_equal(got[:, ~fin], want[:, ~fin].astype(np.float32))
            g, w = got[:, fin], want[:, fin]
            real = np.isfinite(w).all(axis=1)
            assert not np.isfinite(g[~real]).any()  # (an infinite weight's low part is NaN there)
            # 2e-6 of the terms' magnitude (negative weights cancel)
            with np.errstate(invalid="ignore"):
                size = np.abs(P) @ np.abs(V[:, fin]) / np.where(P.sum(1) > 0.0, P.sum(1), 1.0)[:, None]
            assert (np.abs(g - w)[real] <= 2e-6 * np.maximum(1.0, size[real])).all()
