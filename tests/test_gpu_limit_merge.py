"""The clamps of the SA variable after the update, with the flow limiter on (the clamp to SAmin runs
in the repair kernel, the final vt clamp has nothing to do) and off (the final vt clamp alone):
states with negative SA values against the oracle, every iteration."""
import numpy as np
import pytest

from test_gpu_parity import state_err

pytestmark = pytest.mark.gpu


def negative_sa(U):
    rng = np.random.default_rng(5)
    m = rng.random(U.shape[:3]) < 0.2
    U[..., 5] = np.where(m, -np.abs(U[..., 5]) * 0.3 - 1e-9, U[..., 5])
    return U


@pytest.mark.parametrize("limit", [0, 1])
def test_sa_clamps_match_oracle(gpu, oracle, limit):
    from ocfd_b200 import cases
    p, case = cases.airfoil(ni=33, nj=13, scheme=5, flux=4, iflag_limit_flow=limit)
    o, g = oracle.OracleCase(p, case), gpu.Solver(p, case)
    for s in (o, g):
        s.advance(1)
        s.set_state(0, negative_sa(s.get_state(0)))
    for it in range(3):
        o.advance(1)
        g.advance(1)
        np.testing.assert_allclose(g.residual()[1][:6], o.residual()[1][:6], rtol=1e-11, err_msg="step %d" % it)
    assert state_err(o, g) <= 1e-11
    g.close()
    o.close()
