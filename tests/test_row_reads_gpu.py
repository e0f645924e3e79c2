"""Carry-row reads of the DC-EGM continuation by a whole warp (one window of 64
nodes for its 32 queries) against the oracle: savings grids shorter than the
window, around it, not a multiple of a warp (the last warp of a row straddles
two rows and reads lane by lane), and rows so dense in constrained points that
a warp's queries span more nodes than the window.  Bar 1e-10 as in
test_dcegm_gpu (the inversion and crossing chains amplify last-bit differences
of fused multiply-adds)."""

import pytest

from oracle.dcegm import solve as oracle_solve
from pylcm_b200 import examples as E
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taste", [None, 0.05])
@pytest.mark.parametrize("n_savings,n_wealth,n_constrained", [(20, 50, 20), (64, 64, 20), (65, 40, 1), (200, 33, 20),
                                                              (64, 50, 300)])
def test_solve_matches_oracle(n_savings, n_wealth, n_constrained, taste):
    model = E.dcegm_model(4, n_savings, n_wealth, taste=taste is not None, n_constrained=n_constrained)
    params = E.dcegm_params(seed=n_savings, taste_scale=taste)
    V = model.solve(params=params, log_level="off")
    Vo, _ = oracle_solve(model, params)
    for p in Vo:
        for r in Vo[p]:
            assert rel_err(V[p][r], Vo[p][r]) < 1e-10, (p, r)
