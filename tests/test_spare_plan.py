"""Solves and simulations that take over the plan of an earlier call give what
a plan of their own gives, bit for bit; scalar key splits equal the array ones."""

import gc
import threading

import numpy as np
import pytest

from pylcm_b200 import engine as E
from pylcm_b200 import jaxrng
from tests import models as M


@pytest.mark.parametrize("n", [1, 2, 3, 7])
def test_split_key_equals_split(n):
    for k in np.random.default_rng(n).integers(0, 2**32, (50, 2), dtype=np.uint64).astype(np.uint32):
        np.testing.assert_array_equal(jaxrng.split_key(k, n), jaxrng.split(k[None], n)[0])


def _params(k):
    return M.stochastic_params(beta=0.9 + 0.02 * k, crra=1.5 + 0.25 * k)


def _own(model, params, precision):
    return E.SolveEngine(model, precision).solve(params)


def _same(V, want):
    for p in want:
        for r in want[p]:
            np.testing.assert_array_equal(V[p][r], want[p][r].cpu().numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_solves_after_one_another(precision):
    model = M.stochastic_model(5, 40, 60)
    kept = []
    for k in (0, 1, 2, 1):
        V, pol = model.solve(params=_params(k), log_level="off", precision=precision, return_policy=True)
        kept.append((V, pol, *_own(model, _params(k), precision)))
        dev = model.solve(params=_params(3 - k), log_level="off", precision=precision, return_device=True)
        kept.append((dev, None, _own(model, _params(3 - k), precision)[0], None))
    assert model.engine(precision)._spare is not None
    for V, pol, Vw, polw in kept:  # results of earlier calls are untouched by the later ones
        if pol is None:
            V = {p: {r: v.cpu().numpy() for r, v in d.items()} for p, d in V.items()}
        else:
            _same(pol, polw)
        _same(V, Vw)


@pytest.mark.gpu
def test_simulations_after_solves_and_refused_calls():
    model = M.stochastic_model(5, 40, 60)
    rng = np.random.default_rng(0)
    ic = {"wealth": rng.uniform(1, 60, 65), "income": rng.normal(0, 0.25, 65), "regime_id": np.zeros(65, dtype=int)}
    args = dict(initial_conditions=ic, log_level="off", seed=4)
    V0 = model.solve(params=_params(0), log_level="off")
    model.solve(params=_params(2), log_level="off")
    a = model.simulate(params=_params(0), period_to_regime_to_V_arr=V0, **args)
    with pytest.raises(Exception):
        model.solve(params={}, log_level="off")
    b = model.simulate(params=_params(0), **args)
    fresh = M.stochastic_model(5, 40, 60).simulate(params=_params(0), **args)
    for p in a.periods:
        for x in (b, fresh):
            np.testing.assert_array_equal(a.periods[p]["value"], x.periods[p]["value"])
            for g in ("states", "actions"):
                for k in a.periods[p][g]:
                    np.testing.assert_array_equal(a.periods[p][g][k], x.periods[p][g][k])


@pytest.mark.gpu
def test_threads_streams_and_the_limit():
    import torch

    model = M.stochastic_model(5, 40, 60)
    want = {k: _own(model, _params(k), "fp64")[0] for k in range(4)}
    bad = []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream() if k % 2 else torch.cuda.default_stream()):
                for _ in range(5):
                    _same(model.solve(params=_params(k), log_level="off"), want[k])
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
    models = [M.stochastic_model(3, 20, 20) for _ in range(E.SPARE_PLANS + 3)]
    for m in models:
        m.solve(params=_params(0), log_level="off")
    assert sum(m.engine("fp64")._spare is not None for m in models) == E.SPARE_PLANS
    del models, m
    gc.collect()
    assert all(r() is None for r in E._spare_engines)
