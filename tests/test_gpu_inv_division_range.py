"""The FP64 WENO5 / MUSCL3 + Roe fluxes at the top of their reciprocal division's range: one cell
scaled by powers of two around those at which a denominator passes 2^1022, where its reciprocal is
flushed to zero (MUSCL3 squares a difference, 2^511; WENO5 takes its fourth power, 2^255).  The
specialised instantiation of a solve alone must give the residual of the general one, which divides
plainly, everywhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme,powers", [(5, [253.0, 255.5, 257.0, 509.5, 510.4, 511.0, 511.4, 511.9, 512.5, 513.5]),
                                           (7, [253.0, 254.5, 254.8, 255.0, 255.2, 255.5, 256.0, 511.4])])
def test_near_the_largest_denominator(gpu, scheme, powers):
    from meshes import wavy_box
    from ocfd_b200.params import make_params

    def par(s):
        return make_params(ma=0.5, aoa=1.0, if_viscous=0, iflag_scheme=s, iflag_flux=4, cfl=1.0)

    case = wavy_box(15, 12, 9)
    a = gpu.Solver(par(scheme), case)
    b = gpu.Batch([(par(scheme), case), (par(4), case)])
    rng = np.random.default_rng(11)
    shape = a.state_shape(0)
    u0 = np.ones(shape)
    u0[..., 2:4] = 0.1 * rng.standard_normal(shape[:3] + (2,))
    u0[..., 4] = 8.0 + 0.3 * rng.standard_normal(shape[:3])
    u0 *= 1 + 0.05 * rng.standard_normal(shape)
    for q in powers:
        u = u0.copy()
        u[6, 6, 7] *= 2.0 ** q
        u[7, 8, 10, 0] = 2.0 ** q      # alone: a huge density, so a cold and slow cell
        res = []
        for s in (a, b):
            s.set_state(0, u)
            s.compute_residual()
            res.append(s.get_array(0, "Res")[0])
        assert np.array_equal(res[0], res[1], equal_nan=True), q
    a.close()
    b.close()
