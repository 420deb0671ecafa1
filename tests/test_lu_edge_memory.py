"""The edge words of the version-5 sweep are taken, and counted in the footprint, only by handles that run
it: not by explicit schemes, nor where a switch selects another form of the sweep."""
import os

import numpy as np
import pytest

SWITCHES = ("OCFD_LU_V2", "OCFD_LU_V3", "OCFD_LU_V4", "OCFD_LU_V5", "OCFD_LU_TC", "OCFD_LUSGS_PLANES", "OCFD_NO_AUTOTUNE",
            "OCFD_LU_ONE_LAUNCH")


def setup(time, nk=9):
    from meshes import wavy_box
    from ocfd_b200.params import make_params
    raw = dict(ma=0.5, aoa=1.0, if_viscous=0, iflag_scheme=5, iflag_flux=4, time_method=time, cfl=0.5)
    if time == -1:
        raw.update(dt_global=0.1, step_inner_limit=2, res_inner_limit=1e-14)
    return make_params(**raw), wavy_box(101, 65, nk)


def footprint(time, env, monkeypatch, nk=9):
    from ocfd_b200 import build, capi
    if not os.path.exists(capi.LIB_PATH):
        build.build()
    for k in SWITCHES:
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    p, case = setup(time, nk)
    return capi.footprint(p, case)


def edge_bytes(nk, tc):
    TK = 2 if nk <= 3 else (4 if nk <= 5 or tc == 32 else 8)
    TJ = tc // TK
    tiles = -(-64 // TJ) * -(-(nk - 1) // TK)
    return 8 * 5 * (TJ + TK) * tiles * (100 + TJ + TK - 2)


@pytest.mark.parametrize("nk", [3, 5, 9])
def test_footprint_counts_them_where_version_5_runs(monkeypatch, nk):
    none = footprint(0, {"OCFD_LU_V4": "1"}, monkeypatch, nk)
    for env, tc in (({}, 32), ({"OCFD_LU_TC": "32"}, 32), ({"OCFD_LU_V5": "1"}, 32), ({"OCFD_LU_V5": "1", "OCFD_LU_TC": "64"}, 64)):
        more = footprint(0, env, monkeypatch, nk) - none
        assert abs(more - 1.05 * edge_bytes(nk, tc)) <= 1, env
    for env in ({"OCFD_LU_V2": "1"}, {"OCFD_LU_V3": "1"}, {"OCFD_LU_TC": "64"}, {"OCFD_LUSGS_PLANES": "1"}, {"OCFD_NO_AUTOTUNE": "1"},
                {"OCFD_LU_ONE_LAUNCH": "1"}):
        assert footprint(0, env, monkeypatch, nk) == none, env
    # dual time sweeps, the explicit schemes do not; both keep one and two more copies of the state
    state = 1.05 * 8 * 5 * 108 * 72 * (nk + 7)
    assert abs(footprint(-1, {}, monkeypatch, nk) - none - 2 * state - 1.05 * edge_bytes(nk, 32)) <= 1
    for time in (1, 3):
        assert abs(footprint(time, {}, monkeypatch, nk) - none - state) <= 1


@pytest.mark.gpu
@pytest.mark.parametrize("time", [1, 3])
def test_an_explicit_handle_can_sweep_all_the_same(gpu, monkeypatch, time):
    """ocfd_compute_residual with the sweeps, on a handle whose steps have none."""
    p, case = setup(time)
    du = []
    for env in ({}, {"OCFD_LUSGS_PLANES": "1"}):
        for k in SWITCHES:
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        s = gpu.Solver(p, case)
        s.advance(2)
        s.compute_residual(True)
        du.append(s.get_array(0, "DU")[0])
        s.residual()
        s.close()
    assert np.array_equal(du[0], du[1])
