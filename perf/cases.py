"""The workloads whose speed matters to a user of this framework, each through the public binding
(ocfd_b200.capi): solver iterations of single cases and batches, monitors, and the residual of a
given state.

A pass of an iterated case is what a driver's main loop does between two prints: advance a number
of steps, read the residual norms and the force coefficients, take the state to (pinned) host
memory as a checkpoint writer does.  A pass of a residual case is one evaluation for a caller that
owns the state (a verification or an outer Newton / adjoint code): hand the state over, evaluate,
read the residual and its norms.

The norms, forces and residuals of the mixed form are sums and differences of FP32 fluxes that the
C-ABI widens to double; they are kept here in the precision they carry (float32).  The state is FP64
in both forms.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "opencfd-ec_b200"))

from ocfd_b200 import capi, cases as C  # noqa: E402
from ocfd_b200.params import make_params  # noqa: E402

WARM_STEPS = 10  # steps a prepared solve has behind it: the boundary layer has begun to form


def listed():
    return [
        # residual of a given state: an outer code drives the solver, small and ordinary sizes, and
        # both precisions; one block of the Euler channel
        dict(name="residual_fp64_65x33x9", kind="residual", ni=65, nj=33, nk=9, scheme=5, flux=4, prec=0),
        dict(name="residual_mixed_129x65x17", kind="residual", ni=129, nj=65, nk=17, scheme=7, flux=4, prec=1),
        # one airfoil iterated with monitors after every step: the smallest call, latency and launches
        dict(name="foil_sa_fp64_129x33", kind="foil", ni=129, nj=33, scheme=7, flux=4, turb=2, prec=0, time=0, cfl=5.0, steps=1),
        # a coarse wing, 8 small blocks (8320 cells): a grid-convergence study's first level
        dict(name="wing_fp64_41x17x14", kind="wing", ni=41, nj=17, nkw=9, nkt=6, icut=9, scheme=7, prec=0, steps=10),
        # the plain Euler channel (config 1), implicit
        dict(name="bump_fp64_129x65x17", kind="bump", ni=129, nj=65, nk=17, prec=0, time=0, cfl=5.0, steps=20),
        # a time-accurate run of the same channel: dual time stepping, 10 inner iterations per step
        dict(name="bump_dual_97x49x13", kind="bump", ni=97, nj=49, nk=13, prec=0, time=-1, cfl=5.0, steps=2),
        # a k-omega SST airfoil, odd sizes
        dict(name="foil_sst_fp64_257x71", kind="foil", ni=257, nj=71, scheme=5, flux=4, turb=3, prec=0, time=0, cfl=1.0, steps=10),
        # an explicit (RK3) laminar airfoil
        dict(name="foil_lam_rk3_fp64_193x65", kind="foil", ni=193, nj=65, scheme=5, flux=5, turb=0, prec=0, time=3, cfl=0.5, steps=10),
        # the swept wing of config 2 (8 uneven blocks, 2.09 M cells, SA, WENO5 + Roe): the benchmark
        # workload, in both precisions
        dict(name="wing_fp64_257x97x86", kind="wing", ni=257, nj=97, nkw=61, nkt=26, icut=49, scheme=7, prec=0, steps=10),
        dict(name="wing_mixed_257x97x86", kind="wing", ni=257, nj=97, nkw=61, nkt=26, icut=49, scheme=7, prec=1, steps=10),
        # 64 airfoils of different sizes in one handle (config 4): a design sweep's batch
        dict(name="batch_mixed_64", kind="batch", n=64, nseed=1234, prec=1, steps=20),
        # the wing-body of config 3 (24 blocks, 7.8 M cells, SST, MUSCL3), mixed: the largest solve
        dict(name="wingbody_mixed_449x129x137", kind="wingbody", ni=449, nj=129, nkw=97, nkt=41, icut=86, jc1=33, jc2=73,
             prec=1, time=0, cfl=1.0, steps=10),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["residual", "foil", "foil", "wing", "wing", "bump", "batch", "wingbody"])
    prec = rng.randint(0, 1)
    if kind == "residual":
        return dict(kind=kind, ni=_logint(rng, 17, 160), nj=_logint(rng, 12, 80), nk=rng.randint(9, 24), scheme=rng.choice([5, 7]),
                    flux=rng.choice([4, 5]), prec=prec)
    if kind == "foil":
        turb, time = rng.choice([(2, 0), (2, 0), (3, 0), (0, 0), (0, 3)])
        # SST runs at CFL 1 and the explicit scheme at 0.5, which hold from freestream on these meshes
        return dict(kind=kind, ni=2 * _logint(rng, 32, 192) + 1, nj=_logint(rng, 17, 97), scheme=rng.choice([4, 5, 7]),
                    flux=rng.choice([4, 5, 6]), turb=turb, prec=prec, time=time, cfl=0.5 if time == 3 else (1.0 if turb == 3 else 5.0),
                    steps=rng.choice([1, 5, 10]))
    if kind == "wing":
        ni = 4 * rng.randint(10, 64) + 1
        return dict(kind=kind, ni=ni, nj=_logint(rng, 17, 97), nkw=_logint(rng, 9, 61), nkt=_logint(rng, 6, 26), icut=max(9, ni // 5),
                    scheme=rng.choice([5, 7]), prec=prec, steps=rng.choice([5, 10]))
    if kind == "bump":
        time = rng.choice([0, 0, -1])
        return dict(kind=kind, ni=_logint(rng, 33, 257), nj=_logint(rng, 17, 97), nk=_logint(rng, 5, 33), prec=prec, time=time,
                    cfl=5.0, steps=2 if time == -1 else rng.choice([5, 20]))
    if kind == "batch":
        return dict(kind=kind, n=_logint(rng, 2, 64), nseed=rng.randint(1, 9999), prec=prec, steps=rng.choice([5, 10]))
    ni = 2 * rng.randint(40, 150) + 1
    nj = rng.randint(33, 97)
    return dict(kind=kind, ni=ni, nj=nj, nkw=_logint(rng, 13, 65), nkt=_logint(rng, 8, 33), icut=max(12, ni // 5), jc1=nj // 4,
                jc2=(9 * nj) // 16, prec=prec, time=0, cfl=1.0, steps=5)


# ---- the meshes: functions of the sizes alone, made once per process -------------------------
@functools.lru_cache(maxsize=4)
def _mesh(kind, *a):
    if kind == "bump":
        ni, nj, nk = a
        return C.meshgen.channel_bump(ni, nj, nk)
    if kind == "foil":
        ni, nj = a
        return C.airfoil(ni=ni, nj=nj)[1]
    if kind == "wing":
        ni, nj, nkw, nkt, icut = a
        return C.config2(ni=ni, nj=nj, nk_wing=nkw, nk_tip=nkt, i_cut=icut)[1]
    if kind == "batch":
        n, nseed = a
        return [c for _, c in C.config4_batch(n=n, seed=nseed)]
    ni, nj, nkw, nkt, icut, jc1, jc2 = a
    return C.config3(ni=ni, nj=nj, nk_wing=nkw, nk_tip=nkt, i_cut=icut, j_cuts=(jc1, jc2))[1]


def _mesh_of(c):
    k = c["kind"]
    if k in ("bump", "residual"):
        return _mesh("bump", c["ni"], c["nj"], c["nk"])
    if k == "foil":
        return _mesh("foil", c["ni"], c["nj"])
    if k == "wing":
        return _mesh("wing", c["ni"], c["nj"], c["nkw"], c["nkt"], c["icut"])
    if k == "batch":
        return _mesh("batch", c["n"], c["nseed"])
    return _mesh("wingbody", c["ni"], c["nj"], c["nkw"], c["nkt"], c["icut"], c["jc1"], c["jc2"])


def _params(c, rng, mesh=None):
    """The flow of one solve; the seed picks the point of the polar (Mach number and angle)."""
    k = c["kind"]
    dm, da = rng.uniform(-0.02, 0.02), rng.uniform(-0.5, 0.5)
    if k in ("bump", "residual"):
        raw = dict(ma=0.5 + dm, aoa=0.0, if_viscous=0, iflag_scheme=c.get("scheme", 5), iflag_flux=c.get("flux", 4),
                   time_method=c.get("time", 0), cfl=c.get("cfl", 5.0), precision=c["prec"])
        if c.get("time", 0) == -1:
            raw.update(dt_global=0.1, step_inner_limit=10, res_inner_limit=1e-14)
    elif k == "foil":
        raw = dict(ma=0.7 + dm, aoa=2.0 + da, re=6.0e6 if c["turb"] else 5.0e3, if_viscous=1, iflag_turbulence_model=c["turb"],
                   iflag_scheme=c["scheme"], iflag_flux=c["flux"], time_method=c["time"], cfl=c["cfl"], precision=c["prec"],
                   ref_s=0.1)
        if c["turb"] == 3:
            raw.update(kt_inf=1e-8, wt_inf=1e-5)
    elif k == "wing":
        raw = dict(ma=0.8 + dm, aoa=3.0 + da, re=1.0e7, if_viscous=1, iflag_turbulence_model=2, iflag_scheme=c["scheme"],
                   iflag_flux=4, time_method=0, cfl=5.0, precision=c["prec"], ref_s=C.meshgen.wing_ref_area())
    elif k == "batch":
        raw = dict(ma=float(rng.uniform(0.3, 0.85)), aoa=float(rng.uniform(-2.0, 6.0)), re=6.0e6, if_viscous=1,
                   iflag_turbulence_model=2, iflag_scheme=5, iflag_flux=6, time_method=0, cfl=5.0, precision=c["prec"], ref_s=0.1)
    else:
        raw = dict(ma=0.75 + dm, aoa=2.0 + da, re=3.0e6, if_viscous=1, iflag_turbulence_model=3, iflag_scheme=5, iflag_flux=4,
                   time_method=c["time"], cfl=c["cfl"], precision=c["prec"], kt_inf=1e-8, wt_inf=1e-5,
                   ref_s=C.meshgen.wing_ref_area())
    return make_params(**raw)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _given_state(c, seed):
    """A smooth subsonic flow over the whole ghost box of the channel block, U(k, j, i, m)."""
    rng = np.random.default_rng(seed)
    p = _params(c, rng)
    n = (c["nk"] + 7, c["nj"] + 7, c["ni"] + 7)
    z, y, x = np.meshgrid(*[np.linspace(0.0, 1.0, m) for m in n], indexing="ij")

    def wave(amp):
        s = np.zeros(n)
        for _ in range(3):
            a = rng.uniform(2.0, 9.0, 3)
            s += amp / 3.0 * np.sin(a[0] * x + a[1] * y + a[2] * z + rng.uniform(0.0, 2 * np.pi))
        return s

    d = 1.0 + wave(0.08)
    u, v, w = 1.0 + wave(0.1), wave(0.1), wave(0.1)
    pr = (1.0 + wave(0.08)) / (p.gamma * p.ma ** 2)
    U = np.stack([d, d * u, d * v, d * w, pr / (p.gamma - 1.0) + 0.5 * d * (u * u + v * v + w * w)], axis=-1)
    return p, np.ascontiguousarray(U)


def prepare(case, seed):
    c = case
    if c["kind"] == "residual":
        p, U = _given_state(c, seed)
        s = capi.Solver(p, _mesh_of(c))
        pin = _pinned(U.shape)
        pin[...] = U
        return dict(c=c, s=s, U=pin)
    rng = np.random.default_rng(seed)
    if c["kind"] == "batch":
        s = capi.Batch([(_params(c, rng), m) for m in _mesh_of(c)])
    else:
        s = capi.Solver(_params(c, rng), _mesh_of(c))
    s.advance(WARM_STEPS if c.get("time", 0) != -1 else 1)
    # one pinned checkpoint buffer, the blocks one after the other
    shapes = [s.state_shape(b) for b in range(s.nblk)]
    pin = _pinned(sum(math.prod(n) for n in shapes))
    ends = np.cumsum([math.prod(n) for n in shapes])
    out = [pin[e - math.prod(n):e].reshape(n) for n, e in zip(shapes, ends)]
    s.synchronize()
    return dict(c=c, s=s, pin=pin, out=out)


def run(state):
    c, s = state["c"], state["s"]
    as_computed = np.float32 if c["prec"] else np.float64
    if c["kind"] == "residual":
        s.set_state(0, state["U"])
        s.compute_residual()
        rmax, rrms = s.residual()
        res = s.get_array(0, "Res")[0]
        return dict(res=res.astype(as_computed, copy=False), rmax=rmax.astype(as_computed), rrms=rrms.astype(as_computed))
    s.advance(c["steps"])
    rmax, rrms = s.residual_all()
    ft, cl, cd, cs = s.forces_all()
    for b, o in enumerate(state["out"]):
        s.get_state(b, o)
    return dict(U=state["pin"], rmax=rmax.astype(as_computed), rrms=rrms.astype(as_computed), ft=ft.astype(as_computed),
                cl=cl.astype(as_computed), cd=cd.astype(as_computed), cs=cs.astype(as_computed))


def _cells(c):
    m = _mesh_of(c)
    return sum(x.ncells for x in m) if isinstance(m, list) else m.ncells


def work(case):
    """Bytes: per step, one pass of the residual (state and metrics in, residual, dt and spectral
    radii out) and one of each LU-SGS sweep (they cannot start before it is done), or one residual
    and update pass per RK3 stage, plus the state handed over.  Operations: additions,
    multiplications, divisions and roots of the schemes, counted from their formulas."""
    c = case
    n = _cells(c)
    nv = 5 if c["kind"] in ("bump", "residual") else {0: 5, 2: 6, 3: 7}[c.get("turb", 3 if c["kind"] == "wingbody" else 2)]
    f = 4 if c["prec"] else 8
    visc = c["kind"] not in ("bump", "residual")
    metrics = 54 if visc else 21
    recon = {4: 40, 5: 50, 7: 150}[c.get("scheme", 5)] * 5
    face = recon + 200 + (170 if visc else 0) + 60 * (nv - 5)
    res_b = 8 * nv + f * (metrics + nv + 7)
    if c["kind"] == "residual":
        return dict(bytes=float(n * (2 * 8 * nv + res_b)), flops=float(n * (3 * face + 80)))
    time = c.get("time", 0)
    if time == 3:
        step_b, step_f = 3 * (res_b + f * (nv + 1) + 24 * nv), 3 * (3 * face + 120)
    else:
        sweep = 8 * nv * 2 + f * (7 + 12) + f * nv + 8
        step_b, step_f = res_b + 2 * sweep + 8 * nv, 3 * face + 120 + 2 * (3 * 85 + 40)
    iters = c["steps"] * (10 if time == -1 else 1)
    return dict(bytes=float(n * (iters * step_b + 16 * nv)), flops=float(n * iters * step_f))


# ---- the residual of the Euler channel in 64 bits, plain torch -------------------------------
def _minmod(a, b):
    r = torch.where(a.abs() <= b.abs(), a, b)
    return torch.where(a * b <= 0, torch.zeros_like(a), r)


def _cd2(u):
    m = 0.5 * (u[3] + u[4])
    return m, m


def _muscl2c(u):
    um, u0, u1, u2 = u[2], u[3], u[4], u[5]
    return (u0 + 0.5 * _minmod(u1 - u0, 2 * (u0 - um)), u1 - 0.5 * _minmod(u1 - u0, 2 * (u2 - u1)))


def _muscl3(u):
    ep, k3 = 1e-6, 1.0 / 3.0

    def side(up, um):
        s = (2 * up * um + ep) / (up * up + um * um + ep)
        return s

    up, um = u[4] - u[3], u[3] - u[2]
    s = side(up, um)
    L = u[3] + 0.25 * s * ((1 - k3 * s) * um + (1 + k3 * s) * up)
    up, um = u[5] - u[4], u[4] - u[3]
    s = side(up, um)
    return L, u[4] - 0.25 * s * ((1 - k3 * s) * up + (1 + k3 * s) * um)


def _weno5_side(a, b, c, d, e):
    """Value at the face between c and d, from a, b, c (upwind) and d, e."""
    S0 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    S1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    S2 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    w0, w1, w2 = 0.3 / (1e-6 + S0) ** 2, 0.6 / (1e-6 + S1) ** 2, 0.1 / (1e-6 + S2) ** 2
    q0, q1, q2 = c / 3 + 5 * d / 6 - e / 6, -b / 6 + 5 * c / 6 + d / 3, a / 3 - 7 * b / 6 + 11 * c / 6
    return (w0 * q0 + w1 * q1 + w2 * q2) / (w0 + w1 + w2)


def _weno5(u):
    return _weno5_side(u[1], u[2], u[3], u[4], u[5]), _weno5_side(u[6], u[5], u[4], u[3], u[2])


def _roe(l, r, g):
    dl, ul, vl, wl, pl = l
    dr, ur, vr, wr, pr = r
    kl, kr = ul * ul + vl * vl + wl * wl, ur * ur + vr * vr + wr * wr
    hl, hr = g * pl / ((g - 1) * dl) + 0.5 * kl, g * pr / ((g - 1) * dr) + 0.5 * kr
    Ul = [dl, dl * ul, dl * vl, dl * wl, pl / (g - 1) + 0.5 * dl * kl]
    Ur = [dr, dr * ur, dr * vr, dr * wr, pr / (g - 1) + 0.5 * dr * kr]
    Fl = [Ul[1], Ul[1] * ul + pl, Ul[2] * ul, Ul[3] * ul, ul * (Ul[4] + pl)]
    Fr = [Ur[1], Ur[1] * ur + pr, Ur[2] * ur, Ur[3] * ur, ur * (Ur[4] + pr)]
    t = torch.sqrt(dr / dl)
    u, v, w, h = [(a + t * b) / (1 + t) for a, b in ((ul, ur), (vl, vr), (wl, wr), (hl, hr))]
    q = u * u + v * v + w * w
    a = torch.sqrt((g - 1) * (h - 0.5 * q))
    fix = lambda x: torch.where(x < 0.1, (x * x + 0.01) / 0.2, x)  # noqa: E731
    l1, l2, l3 = fix((u - a).abs()), fix(u.abs()), fix((u + a).abs())
    e8 = float(np.float32(1e-8))
    dd = dr - dl
    a2 = (Ur[2] - Ul[2]) / (v + e8) - dd
    a3 = (Ur[3] - Ul[3]) / (w + e8) - dd
    a4 = (g - 1) * (dd * (h - q) + u * (Ur[1] - Ul[1]) + v * (Ur[2] - Ul[2]) + w * (Ur[3] - Ul[3]) - (Ur[4] - Ul[4])) / (a * a)
    a1 = ((u + a) * dd - Ur[1] + Ul[1] - a * a4) / (2 * a)
    a5 = dd - (a1 + a4)
    D = [l1 * a1 + l2 * a4 + l3 * a5,
         l1 * a1 * (u - a) + l2 * a4 * u + l3 * a5 * (u + a),
         l1 * a1 * v + l2 * a2 * v + l2 * a4 * v + l3 * a5 * v,
         l1 * a1 * w + l2 * a3 * w + l2 * a4 * w + l3 * a5 * w,
         l1 * a1 * (h - u * a) + l2 * a2 * v * v + l2 * a3 * w * w + l2 * a4 * 0.5 * q + l3 * a5 * (h + u * a)]
    return [0.5 * (Fl[m] + Fr[m]) - 0.5 * D[m] for m in range(5)]


def _van_leer(l, r, g):
    def part(s, sg):
        d, u, v, w, p = s
        a = torch.sqrt(g * p / d)
        M, k = u / a, u * u + v * v + w * w
        full = [d * u, d * u * u + p, d * u * v, d * u * w, u * (g * p / (g - 1) + 0.5 * d * k)]
        t = sg * 0.25 * d * a * (1 + sg * M) ** 2
        b = (g - 1) * u + sg * 2 * a
        half = [t, t * b / g, t * v, t * w, t * (0.5 * b * b / (g * g - 1) + 0.5 * (v * v + w * w))]
        zero = torch.zeros_like(d)
        return [torch.where(sg * M >= 1, full[m], torch.where(M.abs() < 1, half[m], zero)) for m in range(5)]

    return [x + y for x, y in zip(part(l, 1.0), part(r, -1.0))]


def _euler_residual(c, p, U, xyz):
    g = p.gamma
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    U = torch.as_tensor(U, device=dev)
    X = torch.as_tensor(np.ascontiguousarray(xyz.transpose(1, 2, 3, 0)), device=dev)  # nodes (k, j, i, 3)
    d = U[..., 0]
    vel = [U[..., m] / d for m in (1, 2, 3)]
    pr = (g - 1) * (U[..., 4] - 0.5 * d * sum(v * v for v in vel))
    prim = [d] + vel + [pr]
    nx, ny, nz = c["ni"], c["nj"], c["nk"]
    res = [torch.zeros((nz - 1, ny - 1, nx - 1), dtype=torch.float64, device=dev) for _ in range(5)]
    scheme = {5: _muscl3, 7: _weno5}[c["scheme"]]
    flux = {4: _roe, 5: _van_leer}[c["flux"]]

    def node(di, dj, dk):
        return X[dk:, dj:, di:]

    for ax, nd in ((2, nx), (1, ny), (0, nz)):  # i, j, k faces; ax is the array axis of the direction
        # the face's diagonals, cut to the faces of interior cells
        def at(di, dj, dk):
            n = [nz - 1, ny - 1, nx - 1]
            n[ax] = nd
            return node(di, dj, dk)[:n[0], :n[1], :n[2]]
        if ax == 2:
            t1, t2 = at(0, 1, 0) - at(0, 0, 1), at(0, 1, 1) - at(0, 0, 0)
        elif ax == 1:
            t1, t2 = at(1, 0, 1) - at(0, 0, 0), at(1, 0, 0) - at(0, 0, 1)
        else:
            t1, t2 = at(1, 1, 0) - at(0, 0, 0), at(0, 1, 0) - at(1, 0, 0)
        s = torch.linalg.cross(t1, t2)
        ss = torch.linalg.vector_norm(s, dim=-1)
        S, n1 = 0.5 * ss, s / ss[..., None]
        n2 = t1 / torch.linalg.vector_norm(t1, dim=-1)[..., None]
        n3 = torch.linalg.cross(n1, n2)

        def stencil(a):  # cells idx-4 .. idx+3 along the direction, for every face
            a = a[tuple(slice(4, -4) if q != ax else slice(None) for q in range(3))]
            return [a.narrow(ax, q, nd) for q in range(8)]
        idx = torch.arange(1, nd + 1, device=dev).view([-1 if q == ax else 1 for q in range(3)])
        edge, near = (idx == 1) | (idx == nd), (idx < 4) | (idx > nd - 3)
        L, R = [], []
        for a in prim:
            u = stencil(a)
            l, r = scheme(u)
            lb, rb = _muscl2c(u)
            lc, rc = _cd2(u)
            L.append(torch.where(edge, lc, torch.where(near, lb, l)))
            R.append(torch.where(edge, rc, torch.where(near, rb, r)))

        def turn(q):
            v = torch.stack(q[1:4], dim=-1)
            return [q[0], (v * n1).sum(-1), (v * n2).sum(-1), (v * n3).sum(-1), q[4]]
        F = flux(turn(L), turn(R), g)
        mom = F[1][..., None] * n1 + F[2][..., None] * n2 + F[3][..., None] * n3
        F = [F[0], mom[..., 0], mom[..., 1], mom[..., 2], F[4]]
        if ax == 0:  # the symmetry planes of k take the central flux of the averaged state
            q = [0.5 * (u[3] + u[4]) for u in map(stencil, prim)]
            un = q[1] * n1[..., 0] + q[2] * n1[..., 1] + q[3] * n1[..., 2]
            E = q[4] / (g - 1) + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)
            K = [q[0] * un] + [q[0] * un * q[m + 1] + q[4] * n1[..., m] for m in range(3)] + [(E + q[4]) * un]
            F = [torch.where(edge, b, a) for a, b in zip(F, K)]
        for m in range(5):
            f = F[m] * S
            res[m] -= f.narrow(ax, 1, nd - 1) - f.narrow(ax, 0, nd - 1)
    return torch.stack(res, dim=-1)


def exact(case, seed):
    """The residual cases.  The iterated cases have none: a whole solver (two implicit sweeps over
    the cells in order, limiters, boundary conditions, turbulence) many times over is beyond plain
    array code in the time there is."""
    c = case
    if c["kind"] != "residual":
        return None
    p, U = _given_state(c, seed)
    r = _euler_residual(c, p, U, _mesh_of(c).xyz[0]).cpu().numpy()
    flat = r.reshape(-1, 5)
    rmax, rrms = np.zeros(7), np.zeros(7)
    rmax[:5], rrms[:5] = np.abs(flat).max(0), np.sqrt((flat ** 2).mean(0))
    return dict(res=r, rmax=rmax, rrms=rrms)
