"""LU-SGS version 5 (the default sweep): tile edges, remainders and error recovery.

The FP64 form gives the bits of the one-launch-per-hyperplane order, the mixed form the bits of
version 4, on random states over block shapes that end inside a tile, on its edge and one past it,
down to one cell; no tolerance is involved.  A timed-out wait is reported and leaves the handle
usable."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nodes per direction: 1 cell, inside a tile (8 x 4 columns; 16 x 2 for two-cell-thick blocks), its edge, one past it
SHAPES = [(2, 2, 2), (3, 10, 6), (9, 9, 5), (10, 18, 3), (17, 17, 9), (20, 33, 4), (34, 8, 10), (12, 16, 17)]


def make(turb, prec, shape):
    from meshes import wavy_box
    from ocfd_b200.params import make_params
    visc = turb >= 0
    raw = dict(ma=0.5, aoa=3.0, if_viscous=int(visc), iflag_turbulence_model=max(turb, 0), iflag_scheme=5, iflag_flux=4, re=1e4,
               cfl=2.0, precision=prec)
    if turb == 3:
        raw.update(kt_inf=1e-8, wt_inf=1e-5, cfl=1.0)
    return make_params(**raw), wavy_box(*shape)


def du(gpu, p, case, env, seed=3):
    os.environ.update(env)
    try:
        s = gpu.Solver(p, case)
    finally:
        for k in env:
            os.environ.pop(k)
    rng = np.random.default_rng(seed)
    for b in range(s.nblk):
        u = s.get_state(b)
        u *= 1 + 0.02 * rng.standard_normal(u.shape)
        u[..., 1:4] += 0.1 * rng.standard_normal(u[..., 1:4].shape)
        s.set_state(b, u)
    s.compute_residual(True)
    out = [s.get_array(b, "DU")[0] for b in range(s.nblk)]
    ver = s.lu_kernel_version()
    s.close()
    return out, ver


def same(a, b):
    # equal values, NaN where NaN (a zero's sign may differ: the halved products are summed in one order)
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("turb", [-1, 0, 2, 3])
@pytest.mark.parametrize("shape", SHAPES)
def test_fp64_equals_hyperplanes(gpu, turb, shape):
    p, case = make(turb, 0, shape)
    ref, _ = du(gpu, p, case, {"OCFD_LUSGS_PLANES": "1"})
    got, ver = du(gpu, p, case, {})
    assert ver == 5
    assert same(got, ref)
    got64, _ = du(gpu, p, case, {"OCFD_LU_V5": "1", "OCFD_LU_TC": "64"})
    assert same(got64, ref)


@pytest.mark.parametrize("turb", [-1, 0, 2, 3])
@pytest.mark.parametrize("shape", SHAPES[2:])
def test_mixed_equals_version_4(gpu, turb, shape):
    p, case = make(turb, 1, shape)
    ref, _ = du(gpu, p, case, {"OCFD_LU_V4": "1", "OCFD_LU_TC": "32"})
    got, ver = du(gpu, p, case, {})
    assert ver == 5
    for a, b in zip(got, ref):
        # halving the face area and radius first is exact unless a product is subnormal in FP32
        assert np.array_equal(np.where(np.abs(a) < 1e-36, 0, a), np.where(np.abs(b) < 1e-36, 0, b))


def test_operands_outside_the_fast_division(gpu):
    """Densities at the edges of the format (one unit below 1: the reciprocal whose mantissa is all
    ones; very small and very large) take the same bits as the plain division."""
    p, case = make(0, 0, (9, 9, 5))

    def run(env):
        os.environ.update(env)
        try:
            s = gpu.Solver(p, case)
        finally:
            for k in env:
                os.environ.pop(k)
        u = s.get_state(0)
        u[:, :, :, 0] = np.nextafter(1.0, 0.0)
        u[4, 5, 6] *= 2.0 ** -520
        u[5, 6, 7] *= 2.0 ** 515
        s.set_state(0, u)
        s.compute_residual(True)
        d = s.get_array(0, "DU")[0]
        s.close()
        return d

    assert np.array_equal(run({"OCFD_LUSGS_PLANES": "1"}), run({}), equal_nan=True)


def test_timeout_is_reported_and_the_handle_recovers(gpu):
    from ocfd_b200 import cases
    p, case = cases.config2_small()
    ref = gpu.Solver(p, case)
    ref.advance(2)
    os.environ["OCFD_LU_SPIN_LIMIT"] = "0"
    os.environ["OCFD_LU_V5"] = "1"
    try:
        g = gpu.Solver(p, case)
    finally:
        os.environ.pop("OCFD_LU_SPIN_LIMIT")
        os.environ.pop("OCFD_LU_V5")
    assert g.lu_kernel_version() == 5
    g.advance(1)
    with pytest.raises((gpu.OcfdError, FloatingPointError)) as e:
        g.residual()
    if isinstance(e.value, gpu.OcfdError):
        assert e.value.code == gpu.OCFD_ERR_TIMEOUT
    g.close()
    h = gpu.Solver(p, case)
    h.advance(2)
    for b in range(h.nblk):
        assert np.array_equal(h.get_state(b), ref.get_state(b))
    h.close()
    ref.close()
