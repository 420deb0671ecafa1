"""A handle whose LU-SGS sweep timed out goes on after the error is read: the edge words are empty again
and the flag is down, so the next sweep gives the hyperplane-order bits and the next steps a new
handle's.  Until it is read, sweeps change nothing.  (A bound of 0 gives up at the first word that is
not there yet.)"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 4000000


def noisy(s, seed=3):
    rng = np.random.default_rng(seed)
    u = s.get_state(0)
    u *= 1 + 0.02 * rng.standard_normal(u.shape)
    u[..., 1:4] += 0.1 * rng.standard_normal(u[..., 1:4].shape)
    return u


def setup(gpu, turb, prec):
    from meshes import wavy_box
    from test_gpu_lu_v5 import make
    p, _ = make(turb, prec, (4, 4, 4))
    case = wavy_box(24, 42, 34)  # 6 x 9 tiles
    # the hyperplane order in FP64; the mixed form's bits are version 4's
    env = {"OCFD_LU_V4": "1", "OCFD_LU_TC": "32"} if prec else {"OCFD_LUSGS_PLANES": "1"}
    os.environ.update(env)
    try:
        ref = gpu.Solver(p, case)
    finally:
        for k in env:
            os.environ.pop(k)
    s = gpu.Solver(p, case)
    assert s.lu_kernel_version() == 5
    return s, ref, noisy(ref)


def time_out(gpu, s, u):
    s.set_state(0, u)
    s.set_lu_wait_limit(0)
    s.compute_residual(True)
    s.set_lu_wait_limit(LIMIT)


def read_error(gpu, s, reader):
    with pytest.raises(gpu.OcfdError) as e:
        getattr(s, reader)()
    assert e.value.code == gpu.OCFD_ERR_TIMEOUT


@pytest.mark.parametrize("reader", ["residual", "residual_all", "residual_static"])
@pytest.mark.parametrize("turb,prec", [(-1, 0), (0, 0), (0, 1)])
def test_the_same_handle_goes_on(gpu, turb, prec, reader):
    s, ref, u = setup(gpu, turb, prec)
    time_out(gpu, s, u)
    read_error(gpu, s, reader)
    for h in (s, ref):
        h.set_state(0, u)
        h.compute_residual(True)
    assert np.array_equal(s.get_array(0, "DU")[0], ref.get_array(0, "DU")[0])
    getattr(s, reader)()  # and the error is reported once
    for h in (s, ref):
        h.init_flow()
        h.advance(3)
    assert np.array_equal(s.get_state(0), ref.get_state(0))
    s.close()
    ref.close()


def test_nothing_is_swept_until_the_error_is_read(gpu):
    s, ref, u = setup(gpu, 0, 0)
    time_out(gpu, s, u)
    lost = s.get_array(0, "DU")[0]
    s.set_state(0, 1.01 * u)
    s.compute_residual(True)
    assert np.array_equal(s.get_array(0, "DU")[0], lost, equal_nan=True)
    read_error(gpu, s, "residual")
    for h in (s, ref):
        h.set_state(0, u)
        h.compute_residual(True)
    assert np.array_equal(s.get_array(0, "DU")[0], ref.get_array(0, "DU")[0])
    s.close()
    ref.close()


@pytest.mark.parametrize("env", [{}, {"OCFD_LU_V3": "1"}, {"OCFD_LU_V4": "1", "OCFD_LU_TC": "64"}, {"OCFD_LU_V4": "1", "OCFD_LU_ONE_LAUNCH": "1"}])
def test_a_new_limit_keeps_the_sweep_form(gpu, env):
    from ocfd_b200 import cases
    p, case = cases.config2_small()
    os.environ.update(env)
    try:
        s = gpu.Solver(p, case)
    finally:
        for k in env:
            os.environ.pop(k)
    form = s.lu_kernel_version(), s.lu_tile_width(), s.lu_one_launch()
    s.advance(1)
    s.set_lu_wait_limit(LIMIT // 2)
    assert (s.lu_kernel_version(), s.lu_tile_width(), s.lu_one_launch()) == form
    s.advance(1)
    ref = gpu.Solver(p, case)
    ref.advance(2)
    for b in range(s.nblk):
        assert np.array_equal(s.get_state(b), ref.get_state(b))
    with pytest.raises(gpu.OcfdError):
        s.set_lu_wait_limit(-1)
    s.close()
    ref.close()
