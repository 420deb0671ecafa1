"""The sweep that runs without a switch (version 5 on 32-column tiles) on what single small blocks do not
reach: several blocks with cuts inside tiles, dual time's diagonal, and handles with more tiles than the
GPU has SMs on blocks of different lengths, where a CTA takes one tile after another and its slot and
barrier phases carry over.  FP64 against the hyperplane order, bit for bit; mixed against version 4 on
random states, bit for bit where |DU| is 1e-36 or more (below, a product subnormal in FP32 may differ,
as in test_gpu_lu_v5.py)."""
import os

import numpy as np
import pytest

from test_gpu_lu_versions import NAMES, bits_equal, case_list, run

pytestmark = pytest.mark.gpu

V4 = {"OCFD_LU_V4": "1", "OCFD_LU_TC": "32"}


def sweep_noisy(gpu, make_handle, env, amp):
    """DU of every block after two residuals with the sweeps (the second meets the first one's buffers) of a
    random state; the kernel version."""
    os.environ.update(env)
    try:
        s = make_handle()
    finally:
        for k in env:
            os.environ.pop(k)
    rng = np.random.default_rng(5)
    for b in range(s.nblk):
        u = s.get_state(b)
        u *= 1 + 0.02 * rng.standard_normal(u.shape)
        u[..., 1:4] += amp * rng.standard_normal(u[..., 1:4].shape)
        s.set_state(b, u)
    for _ in range(2):
        s.compute_residual(True)
    du = [s.get_array(b, "DU")[0] for b in range(s.nblk)]
    ver = s.lu_kernel_version()
    s.close()
    assert all(np.isfinite(x).all() for x in du)
    return du, ver


def same_du(a, b, mixed):
    if not mixed:
        return all(np.array_equal(x, y) for x, y in zip(a, b))
    return all(np.array_equal(np.where(np.abs(x) < 1e-36, 0, x), np.where(np.abs(y) < 1e-36, 0, y)) for x, y in zip(a, b))


@pytest.mark.parametrize("name", NAMES)
def test_default_sweep_over_three_steps(gpu, name):
    p, case = case_list()[name]
    refU, refDU, _, _ = run(gpu, p, case, {"OCFD_LUSGS_PLANES": "1"}, 3)
    U, DU, v, t = run(gpu, p, case, {}, 3)
    assert (v, t) == (5, 32)
    assert bits_equal(U, refU)
    assert same_du(DU, refDU, False)


@pytest.mark.parametrize("name", NAMES)
def test_default_mixed_sweep_of_several_blocks(gpu, name):
    p, case = case_list()[name]
    p = p.copy()
    p.precision = 1
    ref, _ = sweep_noisy(gpu, lambda: gpu.Solver(p, case), V4, 0.05)
    got, ver = sweep_noisy(gpu, lambda: gpu.Solver(p, case), {}, 0.05)
    assert ver == 5
    assert same_du(got, ref, True)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("turb", [0, 2, 3])
def test_more_tiles_than_sms(gpu, turb, prec):
    from meshes import wavy_box
    from test_gpu_lu_v5 import make
    p, _ = make(turb, prec, (4, 4, 4))
    cases = [wavy_box(nx, ny, nz) for nx, ny, nz in [(7, 66, 34), (40, 62, 31), (23, 50, 40), (5, 70, 6)]]
    tiles = sum(-(-(d[1] - 1) // 8) * -(-(d[2] - 1) // 4) for c in cases for d in c.dims)
    import torch
    assert tiles > 1.5 * torch.cuda.get_device_properties(0).multi_processor_count
    ref, _ = sweep_noisy(gpu, lambda: gpu.Batch([(p, c) for c in cases]), V4 if prec else {"OCFD_LUSGS_PLANES": "1"}, 0.05)
    got, ver = sweep_noisy(gpu, lambda: gpu.Batch([(p, c) for c in cases]), {}, 0.05)
    assert ver == 5
    assert same_du(got, ref, prec)
