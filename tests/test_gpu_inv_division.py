"""The FP64 WENO5 / MUSCL3 + Roe fluxes divide through reciprocals and FMA; the general instantiation
divides plainly.  A batch whose solves use different schemes runs the general one, a solve alone the
specialised one: both must give the same residual bits, on random states, near freestream (densities
one unit below 1, whose reciprocal is the one special case) and with operands outside the range of
the reciprocal form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def states(shape):
    rng = np.random.default_rng(7)
    u = np.ones(shape)
    u[..., 1] = 1.0
    u[..., 2:4] = 0.1 * rng.standard_normal(shape[:3] + (2,))
    u[..., 4] = 8.0 + 0.3 * rng.standard_normal(shape[:3])
    rand = u * (1 + 0.05 * rng.standard_normal(shape))
    free = np.ones(shape)
    free[..., 2:4] = 0.0
    free[..., 4] = 9.0
    free[..., 0] -= rng.integers(0, 3, shape[:3]) * 2.0 ** -53
    free[..., 2] += rng.integers(-1, 2, shape[:3]) * 1e-17
    odd = rand.copy()
    odd[6, 5, 7] *= 2.0 ** -515   # a nearly empty cell
    odd[5, 6, 9] *= 2.0 ** 514
    return {"random": rand, "freestream": free, "out_of_range": odd}


@pytest.mark.parametrize("scheme", [5, 7])
@pytest.mark.parametrize("name", ["random", "freestream", "out_of_range"])
def test_specialised_flux_equals_general(gpu, scheme, name):
    from meshes import wavy_box
    from ocfd_b200.params import make_params

    def par(s):
        return make_params(ma=0.5, aoa=1.0, if_viscous=0, iflag_scheme=s, iflag_flux=4, cfl=1.0)

    case = wavy_box(15, 12, 9)
    a = gpu.Solver(par(scheme), case)
    b = gpu.Batch([(par(scheme), case), (par(4), case)])
    u = states(a.state_shape(0))[name]
    res = []
    for s in (a, b):
        s.set_state(0, u)
        s.compute_residual()
        res.append(s.get_array(0, "Res")[0])
        s.close()
    assert np.array_equal(res[0], res[1], equal_nan=True)
    if name != "out_of_range":
        assert np.isfinite(res[0]).all()
