"""The DC-EGM carry kernel: a warp's last lane reads the node after its own,
which belongs to the next warp.  A value that one thread stores and another may
read at the same time is accessed by relaxed atomics only, and the rules that
complete it leave a completed value as it is, so either gives the same slopes.

CPU: the generated kernel has no other access to the value rows.  GPU: the
stored end slopes are those of the completed rows, for rows that cross warps."""

import re

import numpy as np
import pytest

from pylcm_b200 import examples as E
from pylcm_b200.engine import SolveEngine
from pylcm_b200.solvers import MSSEnvelope
from tests.test_codegen import NVRTC, nvrtc_compile


def _kernel(src: str, name: str) -> str:
    at = src.index(f"{name}(")
    nxt = src.find('extern "C"', at)
    return src[at:nxt if nxt > 0 else len(src)]


@pytest.mark.parametrize("envelope", [None, MSSEnvelope()], ids=["fues", "mss"])
def test_value_rows_are_accessed_by_relaxed_atomics_only(envelope):
    model = E.dcegm_model(4, 40, 50, envelope=envelope)
    eng = SolveEngine(model, "fp64")
    n = 0
    for s in eng.specs:
        if s.terminal or s.solver is None or not hasattr(s.solver, "savings_grid"):
            continue
        rk = eng.egm_kernels(s, eng.targets_at(s, 0), E.dcegm_params(seed=0))
        body = _kernel(rk.src, rk.names()[1])
        assert "lcm_bracket_slopes" in body
        assert len(re.findall(r"lcm_ld_relaxed\(RV \+ ", body)) == 1 and len(re.findall(r"lcm_st_relaxed\(RV \+ ", body)) == 1
        assert not re.search(r"\bRV\s*\[", body)
        if NVRTC.exists():
            rc, log = nvrtc_compile(rk.src)
            assert rc == 0, log[:2000]
        n += 1
    assert n


def _limited(x, f, d):
    h = np.diff(x)
    with np.errstate(all="ignore"):
        delta = np.diff(f) / h
        a, b = np.maximum(d[:-1] / delta, 0.0), np.maximum(d[1:] / delta, 0.0)
        r2 = a * a + b * b
        tau = np.where(r2 > 9.0, 3.0 / np.sqrt(r2), 1.0)
        flat = delta == 0.0
        return np.where(flat, 0.0, tau * a * delta), np.where(flat, 0.0, tau * b * delta)


@pytest.mark.gpu
def test_end_slopes_of_rows_across_warps():
    import torch

    model = E.dcegm_model(4, 150, 60)
    plan = SolveEngine(model, "fp64").plan([E.dcegm_params(seed=k) for k in range(3)])
    for _ in range(3):
        plan.run()
    torch.cuda.synchronize()
    checked = 0
    for b in plan.egm.values():
        rg, rv, mu, nk, es = (b[k].cpu().numpy() for k in ("rg", "rv", "mu", "nk", "es"))
        for slot, i, r in np.ndindex(nk.shape):
            n = min(int(nk[slot, i, r]), b["npad"])
            if n < 2:
                continue
            x, f, d = rg[slot, i, r, :n], rv[slot, i, r, :n], mu[slot, i, r, :n]
            e0, e1 = _limited(x, f, d)
            ok = np.isfinite(f[:-1]) & np.isfinite(f[1:]) & np.isfinite(d[:-1]) & np.isfinite(d[1:]) & (np.diff(x) > 0.0)
            got = es[slot, i, r, : n - 1]
            # (fused multiply-adds in the limiter: a few ulps)
            np.testing.assert_allclose(got[ok, 0], e0[ok], rtol=1e-13, atol=0.0)
            np.testing.assert_allclose(got[ok, 1], e1[ok], rtol=1e-13, atol=0.0)
            assert np.isnan(got[~ok, 0]).all()
            checked += int(ok.sum())
    assert checked > 1000
