"""Kernel (b)'s rows per pass: dealt evenly over the passes, at most 16 (8 where
an odd number of values is held in registers), and the node sum bit for bit at
counts around them."""

import re

import pytest

from pylcm_b200 import examples as E
from pylcm_b200.engine import SolveEngine
from tests.test_expectation_gpu import test_expectation_is_the_node_sum as node_sum


@pytest.mark.parametrize("n,rows", [(7, 7), (9, 5), (12, 12), (13, 7), (16, 16), (17, 9), (24, 12), (33, 11), (48, 16), (49, 13)])
def test_rows_per_pass(n, rows):
    model = E.hc_model(3, 20, 3, n, 10)
    eng = SolveEngine(model, "fp64")
    spec = next(s for s in model.regime_specs if s.name == "alive")
    src = eng.kernels(spec, eng.targets_at(spec, 0), E.hc_params(1, n)).source()
    body = src.split(f"// ---- expectation alive -> alive: K={n} J={n}")[1]
    assert int(re.search(r"double acc\[(\d+)\]", body).group(1)) == rows
    assert rows * -(-n // rows) - n < -(-n // rows)  # fewer idle rows than passes


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 9, 12, 13, 25, 34, 49, 63])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_node_sum(n, precision):
    node_sum(n, precision)
