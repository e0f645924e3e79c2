"""The read of a collapsed row: the search without the line form leaves its
rounding to the compiler (spelled out it is 8 % slower over NaN rows), the line
form spells it out."""

import dataclasses
import re

import pytest

from pylcm_b200.codegen import device_header
from pylcm_b200.engine import SolveEngine, default_config
from tests import models as M


@pytest.mark.parametrize("lanes,read", [(None, "lcm_interp1s"), (2, "lcm_interp1sl")])
def test_read_by_search_form(lanes, read):
    model = M.hc_model(3, 200, 12, 4, 70)
    spec = next(s for s in model.regime_specs if s.name == "alive")
    cfg = None if lanes is None else {"alive": dataclasses.replace(default_config(spec, "fp32"), lanes=lanes)}
    eng = SolveEngine(model, "fp32", configs=cfg)
    rk = eng.kernels(spec, eng.targets_at(spec, 0), M.hc_params(0, 4))
    assert (rk._line is not None) == (lanes is not None)
    body = rk.source().split("lcm_sc1_")[1]
    assert re.search(r"lcm_interp1\w*<", body).group() == read + "<"


def test_collapsed_read_is_not_spelled_out():
    text = device_header()
    body = text.split("T lcm_interp1s(")[1].split("\n}")[0]
    assert "lcm_lerp" not in body and "wl * v0 + wu * v1" in body
    assert "lcm_lerp" in text.split("T lcm_interp1sl(")[1].split("\n}")[0]
