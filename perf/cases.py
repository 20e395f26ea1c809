"""The work that is timed: what users of this library have it do, through its
public entry points.

Three kinds of program use it:

* a parameter study or a request server: meshes live in the batched solver
  (api.Solver), which advances them many iterations per call; the program
  then reads the states back (kind "solve");
* a driver that owns q in pinned host memory and hands it to the solver for
  every iteration (kind "host", ot2d_solver_iterate_host);
* a Fortran-style driver that keeps its own loop and replaces single
  subroutines (routines.*), with its arrays on the device or in host memory
  (kinds "residual" and "implicit").

Sizes are the repository's mesh classes (129x33 ... 769x193) and odd ones
between; flows are its NACA C-mesh cases at subsonic conditions, which keep
running however many passes are made.
"""
import ctypes as C
import math

import numpy as np
import torch

from turns2d_urans_git_gb300 import api, routines as rt
from turns2d_urans_git_gb300.abi import OT2D_FP32_MIXED, OT2D_FP64

CLASSES = ((129, 33), (257, 65), (385, 97), (513, 129), (769, 193))
FOREVER = 1 << 30   # iteration cap of a request that is never retired


def listed():
    return [
        # the parameter study the library is benchmarked on: 64 RANS-SA
        # requests of one mesh size, resident in device memory
        {"name": "mixed_sa_513x129_b64", "kind": "solve", "model": "sa", "precision": "mixed", "jmax": 513,
         "kmax": 129, "batch": 64, "iters": 200},
        # the same batch for a driver that owns every q in host memory
        {"name": "host_mixed_sa_513x129_b64", "kind": "host", "model": "sa", "precision": "mixed", "jmax": 513,
         "kmax": 129, "batch": 64, "iters": 2},
        # a study over airfoils, each on the mesh class that suits it
        {"name": "mixed_sa_classes_b24", "kind": "solve", "model": "sa", "precision": "mixed", "jmax": 0, "kmax": 0,
         "batch": 24, "iters": 200},
        # one small request on its own: the latency of an iteration
        {"name": "mixed_sa_129x33_b1", "kind": "solve", "model": "sa", "precision": "mixed", "jmax": 129, "kmax": 33,
         "batch": 1, "iters": 200},
        # time-spectral pitching requests as the request stream holds them
        {"name": "mixed_ts5_257x65_b4", "kind": "solve", "model": "ts5", "precision": "mixed", "jmax": 257,
         "kmax": 65, "batch": 4, "iters": 100},
        # time-accurate pitching requests, four Newton iterations a step
        {"name": "mixed_pitch_257x65_b16", "kind": "solve", "model": "pitch", "precision": "mixed", "jmax": 257,
         "kmax": 65, "batch": 16, "iters": 96},
        # transonic configuration: k-omega SST, WENO5, ADI line solves
        {"name": "mixed_sst_weno_adi_769x193", "kind": "solve", "model": "sst", "precision": "mixed", "jmax": 769,
         "kmax": 193, "batch": 1, "iters": 50},
        # the plain FP64 path: one inviscid solve ...
        {"name": "fp64_euler_257x65_b1", "kind": "solve", "model": "euler", "precision": "fp64", "jmax": 257,
         "kmax": 65, "batch": 1, "iters": 100},
        # ... and a batch of RANS-SA solves
        {"name": "fp64_sa_385x97_b8", "kind": "solve", "model": "sa", "precision": "fp64", "jmax": 385, "kmax": 97,
         "batch": 8, "iters": 25},
        # a driver that replaces the residual routines, arrays on the device
        {"name": "residual_device_257x65", "kind": "residual", "place": "device", "jmax": 257, "kmax": 65},
        # the same from plain host arrays, on an odd large mesh
        {"name": "residual_host_601x151", "kind": "residual", "place": "host", "jmax": 601, "kmax": 151},
        # a driver that replaces the implicit operator and the SA solve
        {"name": "implicit_device_385x97", "kind": "implicit", "place": "device", "jmax": 385, "kmax": 97},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "host", "residual", "implicit"))
    jmax = 2 * _spread(rng, 40, 300) + 1          # odd, 81 .. 601: an even split of the airfoil
    kmax = min(_spread(rng, 27, 150), jmax // 2)
    if kind in ("residual", "implicit"):
        return {"kind": kind, "place": rng.choice(("device", "host")), "jmax": jmax, "kmax": kmax}
    most = max(1, 2_000_000 // (jmax * kmax))     # cells of the batch
    if kind == "host":
        batch = _spread(rng, 1, min(48, most))
        return {"kind": kind, "model": "sa", "precision": "mixed", "jmax": jmax, "kmax": kmax, "batch": batch,
                "iters": rng.randint(1, 4)}
    model = rng.choice(("sa", "sa", "sa", "euler", "ts3", "pitch", "sst"))
    precision = rng.choice(("mixed", "mixed", "fp64"))
    batch = _spread(rng, 1, max(1, min(48, most // (8 if precision == "fp64" else 1) // (3 if model == "ts3" else 1))))
    return {"kind": kind, "model": model, "precision": precision, "jmax": jmax, "kmax": kmax, "batch": batch,
            "iters": 4 * rng.randint(2, 6)}


# ---- inputs -----------------------------------------------------------------

def _case_of(case, rng):
    """One request: (inputs, params, xv, yv)."""
    model, jmax, kmax = case.get("model", "sa"), case["jmax"], case["kmax"]
    naca, alfa = (0.0, 0.0, 0.12), float(rng.uniform(0.0, 1.0))
    if not jmax:   # a study over airfoils and mesh classes
        jmax, kmax = CLASSES[int(rng.integers(len(CLASSES)))]
        naca = (float(rng.uniform(0, 0.04)), float(rng.uniform(0.3, 0.5)), float(rng.uniform(0.10, 0.15)))
    common = dict(naca=naca, ds_wall=api.wall_spacing(kmax), irhsy=-3, ilim=1, ilhs=1, iconstant_cfl=1, alfa=alfa)
    sa = dict(invisc=0, lamin=0, iturb=1, rey=3e6, vnuinf=3.0)
    if model == "sa":
        return api.cmesh_case(jmax, kmax, dt=20.0, fsmach=0.2, **sa, **common)
    if model == "euler":
        common["ds_wall"] = max(1e-3, common["ds_wall"])
        return api.cmesh_case(jmax, kmax, dt=10.0, fsmach=0.5, invisc=1, lamin=1, **common)
    if model in ("ts3", "ts5"):
        return api.cmesh_case(jmax, kmax, dt=10.0, fsmach=0.3, timespectral=1, nspec=int(model[2:]), rf=0.02,
                              angmax=2.0, xac=0.25, motiontype=1, **sa, **common)
    if model == "pitch":
        return api.config_pitching(jmax, kmax, viscous=True, iturb=1, ntac=2, itnmax=4, dt=0.05, rf=0.1, angmax=1.0,
                                   fsmach=0.3, alfa=alfa, rey=3e6)
    return api.config_c3(jmax, kmax, fsmach=0.5, alfa=3.0 * alfa, ds_wall=common["ds_wall"], dt=0.1)


def _requests(case, seed):
    """The requests of a batch.  Requests on one mesh share its vertices."""
    rng = np.random.default_rng(seed)
    if not case["jmax"]:
        rng = np.random.default_rng(7)            # the airfoils of the study; the seed moves their flows
        moved = np.random.default_rng(seed)
        out = []
        for _ in range(case["batch"]):
            inp, prm, xv, yv = _case_of(case, rng)
            inp.alfa += float(moved.uniform(0.0, 0.5))
            out.append((api.params_from_inputs(inp), xv, yv))
        return out
    return [c[1:] for c in (_case_of(case, rng) for _ in range(case["batch"]))]


def _solver(case, seed):
    # keep_q: the state of a request that failed can still be read
    sv = api.Solver(OT2D_FP32_MIXED if case["precision"] == "mixed" else OT2D_FP64, keep_q=True)
    reqs = _requests(case, seed)
    cap = 4000 if case["model"] == "pitch" else FOREVER   # physical steps of a time-accurate request
    ids = [sv.add(p, xv, yv, orders=0.0, max_iters=cap) for p, xv, yv in reqs]
    return sv, ids, [r[0] for r in reqs]


class _Arrays:
    """The arrays of a driver with one mesh, as the reference's main program
    allocates them: a developed-looking SA state on a NACA C-mesh."""

    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        self.rng = rng
        _, p, xv, yv = api.config_c2(case["jmax"], case["kmax"], fsmach=0.3, alfa=float(rng.uniform(0, 6)), rey=6e6,
                                     ds_wall=api.wall_spacing(case["kmax"]))
        self.p, n2 = p, p.jd * p.kd
        rt.set_params(p)
        z = lambda n=n2: np.zeros(n)  # noqa: E731
        self.xv, self.yv = xv.ravel().copy(), yv.ravel().copy()
        self.x, self.y, self.xx, self.xy, self.yx, self.yy = z(), z(), z(), z(), z(), z()
        self.ug, self.vg, self.tscale, self.bt = z(), z(), z(), np.ones(n2)
        self.ugv, self.vgv = z(self.xv.size), z(self.xv.size)
        self.iblank = np.ones(n2, dtype=np.int32)
        self.q, self.s = z(n2 * p.nq), z(n2 * p.nv)
        rt.find_cellcenter(self.x, self.y, self.xv, self.yv, p.jd, p.kd)
        rt.metfv(self.q, self.x, self.y, self.xv, self.yv, self.xx, self.xy, self.yx, self.yy, p.jd, p.kd)
        # density, velocity and pressure about the freestream, smooth over the mesh
        j, k = np.meshgrid(np.arange(p.jd) / p.jd, np.arange(p.kd) / p.kd)
        f = lambda: sum(rng.uniform(-0.03, 0.03) * np.sin(2 * np.pi * (a * j + b * k + rng.uniform()))  # noqa: E731
                        for a in (1, 2, 5) for b in (1, 3)).ravel()
        q = self.q.reshape(p.nq, n2)
        J = q[p.nq - 1]
        rho, u, v, pr = p.rinf * (1 + f()), p.uinf + 0.3 * f(), p.vinf + 0.3 * f(), p.pinf * (1 + f())
        q[0], q[1], q[2] = rho / J, rho * u / J, rho * v / J
        q[3] = (pr / p.gm1 + 0.5 * rho * (u * u + v * v)) / J
        q[4] = p.vnuinf * 10.0 ** (1.5 + 20 * f())
        self.turmu = 10.0 ** (20 * f())
        self.s0 = 1e-5 * np.concatenate([f() for _ in range(p.nv)])

    def on_device(self):
        for name, a in list(self.__dict__.items()):
            if isinstance(a, np.ndarray):
                setattr(self, name, torch.from_numpy(a).cuda())
        return self


def prepare(case, seed):
    if case["kind"] == "solve":
        return (case,) + _solver(case, seed)
    if case["kind"] == "host":
        sv, ids, prms = _solver(case, seed)
        q = [torch.from_numpy(sv.get_q(i, p)).pin_memory() for i, p in zip(ids, prms)]
        c_ids = (C.c_int32 * len(ids))(*ids)
        c_q = (C.POINTER(C.c_double) * len(ids))(*[C.cast(t.data_ptr(), C.POINTER(C.c_double)) for t in q])
        return case, sv, c_ids, c_q, q
    a = _Arrays(case, seed)
    if case["kind"] == "implicit":
        p = a.p
        rt.time_step(a.q, a.xx, a.xy, a.yx, a.yy, a.ug, a.vg, a.tscale, a.bt, a.iblank, p.jd, p.kd)
    return case, a.on_device() if case["place"] == "device" else a


def run(state):
    kind = state[0]["kind"]
    if kind == "solve":
        case, sv, ids, prms = state
        sv.iterate(case["iters"])
        return [sv.get_q(i, p) for i, p in zip(ids, prms)]
    if kind == "host":
        case, sv, c_ids, c_q, q = state
        rc = api.lib().ot2d_solver_iterate_host(C.c_void_p(sv._h), len(q), c_ids, c_q, case["iters"])
        if rc != 0:
            raise RuntimeError("ot2d_solver_iterate_host failed (%d)" % rc)
        return q
    a = state[1]
    p = a.p
    rt.set_params(p)
    if kind == "residual":
        # the explicit half of a step: time step, s = 0, inviscid and viscous residual
        a.s[:] = 0.0
        rt.time_step(a.q, a.xx, a.xy, a.yx, a.yy, a.ug, a.vg, a.tscale, a.bt, a.iblank, p.jd, p.kd)
        if state[0]["place"] == "device":
            torch.cuda.current_stream().synchronize()   # the library works on its own stream
        rt.rhsup(a.q, a.s, a.xx, a.xy, a.yx, a.yy, a.x, a.y, a.xv, a.yv, a.xv, a.yv, a.xv, a.yv, a.iblank, a.ugv, a.vgv,
                 p.jd, p.kd, 1, 1, a.bt)
        rt.visrhs(a.turmu, a.q, a.s, a.xx, a.xy, a.yx, a.yy, a.ug, a.vg, a.tscale, a.iblank, p.jd, p.kd)
        return {"s": a.s, "tscale": a.tscale}
    # the implicit half: the LU-SGS correction of s, and the SA update of nu_tilde and mu_t
    a.s[:] = a.s0
    if state[0]["place"] == "device":
        torch.cuda.current_stream().synchronize()
    rt.ilu2d(a.q, a.s, p.jd, p.kd, p.jbeg, p.jend, p.kbeg, p.kend, a.xx, a.xy, a.yx, a.yy, a.ug, a.vg, a.turmu, a.tscale)
    rt.vmu_sa(a.q, a.s, a.turmu, a.x, a.y, a.xv, a.yv, a.xx, a.xy, a.yx, a.yy, a.ug, a.vg, p.jd, p.kd, a.tscale,
              a.iblank, 1, 1)
    return {"q": a.q, "s": a.s, "turmu": a.turmu}


# ---- what a pass cannot do without -------------------------------------------

def _cells(case):
    if case["kind"] in ("solve", "host") and not case["jmax"]:
        rng, n = np.random.default_rng(7), 0
        for _ in range(case["batch"]):
            rng.uniform()
            j, k = CLASSES[int(rng.integers(len(CLASSES)))]
            rng.uniform(size=3)
            n += j * k
        return n
    return case["jmax"] * case["kmax"] * case.get("batch", 1)


def work(case):
    n = _cells(case)
    if case["kind"] == "residual":
        # q, metrics, mu_t, vertices and iblank read; s and tscale written
        return {"bytes": n * (6 * 8 + 4 * 8 + 8 + 16 + 4 + 5 * 8 + 8), "flops": n * 900}
    if case["kind"] == "implicit":
        # q, s, metrics, mu_t, tscale, centres and vertices read; q, s, mu_t written
        return {"bytes": n * (6 * 8 + 5 * 8 + 4 * 8 + 16 + 32 + 5 * 8 + 5 * 8 + 8), "flops": n * 700}
    model, r = case["model"], 4 if case["precision"] == "mixed" else 8
    nv = {"euler": 4, "sst": 6}.get(model, 5)
    ns = int(model[2:]) if model[:2] == "ts" else 1
    turb = 0 if model == "euler" else 1
    # per iteration: the FP64 state read and written, the geometry (J, four
    # metrics, iblank, wall distance) read, mu_t read and written
    per = nv * 16 + 5 * r + 4 + turb * 3 * r
    flops = {"euler": 700, "sst": 2600}.get(model, 1700)
    b = n * ns * case["iters"] * per
    if case["kind"] == "host":
        b = n * case["iters"] * (nv * 16 + 5 * r + 4 + 3 * r)
    return {"bytes": b, "flops": n * ns * case["iters"] * flops}


# ---- 64-bit values of the single routines, in numpy ----------------------------

def exact(case, seed):
    """numpy in 64 bits for the single routines.  The solver cases run dozens
    of whole iterations over a batch, minutes of numpy: no value there."""
    if case["kind"] in ("solve", "host"):
        return None
    a = _Arrays(case, seed)
    if case["kind"] == "implicit":
        tscale = _np_time_step(a)
        q, s = _np_ilu2d(a, a.s0, tscale)
        q, turmu = _np_vmu_sa(a, q, s, tscale)
        return {"q": q.ravel(), "s": s.ravel(), "turmu": turmu.ravel()}
    s = _np_rhsup(a) + _np_visrhs(a)
    return {"s": s.ravel(), "tscale": _np_time_step(a).ravel()}


def _grid(a, v):
    """A flat Fortran array as [k, j] (or [n, k, j])."""
    v = np.asarray(v, dtype=np.float64)
    n2 = a.p.jd * a.p.kd
    return v.reshape(a.p.kd, a.p.jd) if v.size == n2 else v.reshape(-1, a.p.kd, a.p.jd)


def _np_prim(a, q=None):
    q = _grid(a, a.q) if q is None else q
    u, v = q[1] / q[0], q[2] / q[0]
    e = q[3] / q[0] - 0.5 * (u * u + v * v)     # internal energy
    return q[-1], u, v, e


def _np_time_step(a):
    _, u, v, e = _np_prim(a)
    c2 = a.p.ggm1 * e
    lam = 0.0
    for mx, my in ((a.xx, a.xy), (a.yx, a.yy)):
        mx, my = _grid(a, mx), _grid(a, my)
        lam = lam + np.abs(u * mx + v * my) + np.sqrt(c2 * (mx * mx + my * my))
    return a.p.h / lam


def _np_roe(gm1, L, R, nx, ny):
    """Roe flux through faces with normal (nx, ny): states (rho, u, v, p)."""
    area = np.hypot(nx, ny)
    nx, ny = nx / area, ny / area
    (rl, ul, vl, pl), (rr, ur, vr, pr) = L, R
    hl = (pl / gm1 + 0.5 * rl * (ul * ul + vl * vl) + pl) / rl
    hr = (pr / gm1 + 0.5 * rr * (ur * ur + vr * vr) + pr) / rr
    w = np.sqrt(rr / rl)
    ra = w * rl
    ua, va, ha = (w * ur + ul) / (w + 1), (w * vr + vl) / (w + 1), (w * hr + hl) / (w + 1)
    c2 = gm1 * (ha - 0.5 * (ua * ua + va * va))
    c = np.sqrt(c2)
    un, unl, unr = nx * ua + ny * va, nx * ul + ny * vl, nx * ur + ny * vr
    cl, cr = np.sqrt(1.0 * gm1 * (hl - 0.5 * (ul * ul + vl * vl))), np.sqrt(gm1 * (hr - 0.5 * (ur * ur + vr * vr)))

    def fixed(lam, dl):   # Harten's entropy fix with the left-to-right spread of the wave speed
        d = 4.0 * dl + 1e-6
        lam = np.abs(lam)
        return np.where(lam <= 0.5 * np.maximum(d, 0.0), lam * lam / d + 0.25 * d, lam)

    l0, lp, lm = fixed(un, unr - unl), fixed(un + c, unr + cr - unl - cl), fixed(un - c, unr - cr - unl + cl)
    dr, du, dv, dp, dun = rr - rl, ur - ul, vr - vl, pr - pl, unr - unl
    b1 = l0 * (dr - dp / c2)
    b2, b3 = lp * (dp + ra * c * dun) / (2 * c2), lm * (dp - ra * c * dun) / (2 * c2)
    b4, b5 = b1 + b2 + b3, c * (b2 - b3)
    b6, b7 = l0 * ra * (du - nx * dun), l0 * ra * (dv - ny * dun)
    d = (b4, ua * b4 + nx * b5 + b6, va * b4 + ny * b5 + b7,
         ha * b4 + un * b5 + ua * b6 + va * b7 - c2 * b1 / gm1)
    f = (rl * unl + rr * unr, rl * ul * unl + rr * ur * unr + nx * (pl + pr),
         rl * vl * unl + rr * vr * unr + ny * (pl + pr), rl * hl * unl + rr * hr * unr)
    return np.stack([0.5 * area * (x - y) for x, y in zip(f, d)])


def _np_muscl(f, n):
    """Third-order MUSCL with the differentiable limiter along the last axis."""
    eps, th, qt = (10.0 / n) ** 3, 1.0 / 3.0, 0.25
    d = np.diff(f, axis=-1)
    m, p = d[..., :-1], d[..., 1:]
    a1 = 3.0 * (p * m + eps)
    phi = qt * a1 / (2.0 * (p - m) ** 2 + a1)
    ql, qr = f.copy(), f.copy()
    ql[..., 1:-1] += phi * ((1 - th) * m + (1 + th) * p)
    qr[..., 1:-1] -= phi * ((1 + th) * m + (1 - th) * p)
    return ql, qr


def _np_rhsup(a):
    p, (J, u, v, e) = a.p, _np_prim(a)
    rho = _grid(a, a.q)[0] * J
    f = np.stack([rho, u, v, p.gm1 * rho * e])
    xv, yv = a.xv.reshape(p.kmax, p.jmax), a.yv.reshape(p.kmax, p.jmax)
    s = np.zeros((p.nv, p.kd, p.jd))
    ql, qr = _np_muscl(f[:, 1:-1, :], p.jmax)
    F = _np_roe(p.gm1, ql[..., :-1], qr[..., 1:], np.diff(yv, axis=0), -np.diff(xv, axis=0))
    s[:4, 1:-1, 1:-1] -= np.diff(F, axis=-1)
    ql, qr = _np_muscl(f[:, :, 1:-1].swapaxes(1, 2), p.kmax)
    F = _np_roe(p.gm1, ql[..., :-1], qr[..., 1:], -np.diff(yv, axis=1).T, np.diff(xv, axis=1).T)
    s[:4, 1:-1, 1:-1] -= np.diff(F, axis=-1).swapaxes(1, 2)
    return s


def _np_laminar(p, e):
    c2b = 198.6 / p.tinf
    t = p.ggm1 * e
    return (c2b + 1.0) * t * np.sqrt(t) / (c2b + t)


def _np_visrhs(a):
    """Thin-layer and cross-derivative viscous terms of both directions."""
    p, (J, u, v, e) = a.p, _np_prim(a)
    turm = _grid(a, a.turmu)
    mu = _np_laminar(p, e)
    vnu, gkap = (mu + turm) * 0.5 / p.rey, (mu + p.pr / 0.9 * turm) * 0.5 / p.rey * p.gamma / p.pr
    xx, xy, yx, yy = (_grid(a, m) for m in (a.xx, a.xy, a.yx, a.yy))
    s = np.zeros((p.nv, p.kd, p.jd))

    def direction(mx, my, ox, oy, U, V, E, G, K, RJ):
        """Along the last axis; (mx, my) this direction's metrics, (ox, oy) the other's."""
        b4 = (mx * mx + my * my) * RJ
        b1, b2, b5 = (b4 + mx * mx / 3 * RJ) * G, (b4 + my * my / 3 * RJ) * G, mx * my / 3 * RJ * G
        b4 = b4 * K
        fa = lambda x: x[:, 1:] + x[:, :-1]  # noqa: E731
        du, dv, de = np.diff(U), np.diff(V), np.diff(E)
        f2 = fa(b1) * du + fa(b5) * dv
        f3 = fa(b5) * du + fa(b2) * dv
        f4 = (fa(U * b1) + fa(V * b5)) * du + (fa(V * b2) + fa(U * b5)) * dv + fa(b4) * de
        # cell terms: products of both directions' metrics at the two side neighbours
        side = lambda x: x[:-2] + x[2:]  # noqa: E731
        c43, c23 = 4.0 / 3.0, -2.0 / 3.0
        d1 = G[1:-1] * side((c43 * mx * ox + my * oy) * RJ)
        d2 = G[1:-1] * side((c43 * my * oy + mx * ox) * RJ)
        d4 = K[1:-1] * side((mx * ox + my * oy) * RJ)
        d5 = G[1:-1] * side((c23 * mx * oy + my * ox) * RJ)
        d7 = G[1:-1] * side((c23 * my * ox + mx * oy) * RJ)
        up, um, vp, vm = U[2:], U[:-2], V[2:], V[:-2]
        dU, dV, dE = 0.5 * (up - um), 0.5 * (vp - vm), 0.5 * (E[2:] - E[:-2])
        return (f2, f3, f4), (d1, d2, d4, d5, d7), (up, um, vp, vm, dU, dV, dE)

    def add(rows, faces, cells):
        """Face differences, and central cell differences (one-sided at the far end)."""
        for n, (f, c) in enumerate(zip(faces, cells)):
            d = np.zeros_like(rows[n])
            d[:, 1:-1] = np.diff(f)
            d[:, 1:-2] += 0.5 * (c[:, 2:-1] - c[:, :-3])
            d[:, -2] += 0.5 * (c[:, -4] - 4 * c[:, -3] + 3 * c[:, -2])
            rows[n] += d

    def cross(d, c):
        (d1, d2, d4, d5, d7), (up, um, vp, vm, dU, dV, dE) = d, c
        f4 = (0.25 * d1 * (up * up - um * um) + 0.25 * d2 * (vp * vp - vm * vm) + 0.5 * d5 * (up + um) * dV +
              0.5 * d7 * (vp + vm) * dU + d4 * dE)
        return d1 * dU + d5 * dV, d7 * dU + d2 * dV, f4

    t = lambda x: x.T.copy()  # noqa: E731
    eta = [t(m) for m in (yx, yy, xx, xy, u, v, e, vnu, gkap, 1 / J)]
    xi = (xx, xy, yx, yy, u, v, e, vnu, gkap, 1 / J)
    for lines, turned in ((eta, True), (xi, False)):   # lines along the last axis
        f, d, c = direction(*lines)
        rows = [np.zeros((f[0].shape[0] - 2, f[0].shape[1] + 1)) for _ in range(3)]
        add(rows, [x[1:-1] for x in f], cross(d, c))
        for n, r in enumerate(rows):
            s[n + 1, 1:-1, 1:-1] += r[:, 1:-1].T if turned else r[:, 1:-1]
    return s


def _np_ilu2d(a, s0, tscale):
    """Two-sweep LU-SGS over the hyperplanes j + k."""
    p, q = a.p, _grid(a, a.q).copy()
    J, u, v, e = _np_prim(a)
    c, H = np.sqrt(p.ggm1 * e), p.gamma * e + 0.5 * (u * u + v * v)
    uv2, rho = 0.5 * (u * u + v * v), q[0] * J
    eps2 = 2.0 * p.epse
    xx, xy, yx, yy = (_grid(a, m) for m in (a.xx, a.xy, a.yx, a.yy))
    rr2 = yx * yx + yy * yy
    vn = 2.0 * rr2 * (p.rmue + _grid(a, a.turmu)) / (p.rey * rho)
    qx, qy, cx, cy = xx * u + xy * v, yx * u + yy * v, c * np.hypot(xx, xy), c * np.sqrt(rr2)
    D = 1.0 / (1.0 + tscale * ((np.abs(qx) + np.abs(qy) + cx + cy) * (1.0 + eps2) + vn))
    s = _grid(a, s0).copy()
    for edge in ((slice(1, -1), 0), (slice(1, -1), -1), (0, slice(1, -1)), (-1, slice(1, -1))):
        s[(slice(0, 4),) + edge] *= D[edge]

    def contribution(k, j, mx, my, qq, cc, vis, sign):
        s1, s2, s3, s4 = s[0, k, j], s[1, k, j], s[2, k, j], s[3, k, j]
        mx, my, qq, cc, uu, vv = mx[k, j], my[k, j], qq[k, j], cc[k, j], u[k, j], v[k, j]
        sp = np.abs(qq) + cc
        chk = 0.5 + 0.5 * np.sign(sign * qq + cc)   # 1 where the wave goes this way
        spec = chk * (qq + sign * sp) + sign * (eps2 * sp + vis[k, j])
        w = chk * (mx * s2 + my * s3 - qq * s1)
        g = chk * p.gm1 * (uv2[k, j] * s1 - (uu * s2 + vv * s3) + s4)
        return np.stack([w + spec * s1, mx * g + uu * w + spec * s2, my * g + vv * w + spec * s3,
                         qq * g + H[k, j] * w + spec * s4])

    zero = np.zeros_like(vn)
    for sign in (1, -1):
        planes = range(2, p.jd + p.kd - 3)
        for m in planes if sign > 0 else reversed(planes):
            j = np.arange(max(1, m - (p.kd - 2)), min(p.jd - 2, m - 1) + 1)
            k = m - j
            t = (contribution(k, j - sign, xx, xy, qx, cx, zero, sign) +
                 contribution(k - sign, j, yx, yy, qy, cy, vn, sign))
            half = 0.5 * tscale[k, j]
            s[:4, k, j] = (s[:4, k, j] + half * t) * D[k, j] if sign > 0 else s[:4, k, j] - half * t * D[k, j]
    return q, s


def _np_turbc(a, q, u, v):
    """nu_tilde on the halo of the C-mesh: far field, wake cut and wall, in the table's order."""
    p, n5 = a.p, q[4]
    yx, yy, xx, xy = (_grid(a, m) for m in (a.yx, a.yy, a.xx, a.xy))
    for b in range(p.nbc):
        js, je, ks, ke = p.jbcs[b], p.jbce[b], p.kbcs[b], p.kbce[b]
        js, je = (p.jmax + x + 1 if x < 0 else x for x in (js, je))
        ks, ke = (p.kmax + x + 1 if x < 0 else x for x in (ks, ke))
        js, ks = js + (js > 1), ks + (ks > 1)
        je, ke = p.jd if je == p.jmax else je, p.kd if ke == p.kmax else ke
        J, K, t, d = slice(js - 1, je), slice(ks - 1, ke), p.ibtyp[b], p.ibdir[b]
        add = 1 if d > 0 else -1
        if t == 5:
            n5[K, J] = -n5[ks - 1 + add, J]
        elif t == 51:
            j = np.arange(js - 1, je)
            jj = p.jd - 1 - j
            n5[ks - 1, j], n5[ks - 1, jj] = n5[ks, jj], n5[ks, j]
        elif t == 47:
            here, inner = ((ks - 1, J), (ks - 1 + add, J)) if abs(d) == 2 else ((K, js - 1), (K, js - 1 + add))
            mx, my = (yx, yy) if abs(d) == 2 else (xx, xy)
            un = add * ((u[here] + u[inner]) * mx[here] + (v[here] + v[inner]) * my[here])
            n5[here] = np.where(un < 0.0, n5[inner], p.vnuinf)
        else:
            raise ValueError("boundary type %d" % t)


def _np_vmu_sa(a, q, s, tscale):
    """One Spalart-Allmaras update: right-hand side, two line solves, mu_t."""
    p = a.p
    J, u, v, e = _np_prim(a, q)
    rho, nul = q[0] * J, _np_laminar(p, e) / (q[0] * J)
    xx, xy, yx, yy = (_grid(a, m) for m in (a.xx, a.xy, a.yx, a.yy))
    cb1, sigma, cb2, kap, cw1, cw2, cw3, cv1 = 0.1355, 0.6666667, 0.622, 0.41, 3.2390678, 0.3, 2.0, 7.1
    _np_turbc(a, q, u, v)
    nt = q[4]
    I = (slice(1, -1), slice(1, -1))  # noqa: E741
    rhs, b = s[4][I].copy(), 0.0
    bands = []
    for ax, mx, my in ((1, xx, xy), (0, yx, yy)):
        lo, hi = ((slice(1, -1), slice(0, -2)), (slice(1, -1), slice(2, None))) if ax else (
            (slice(0, -2), slice(1, -1)), (slice(2, None), slice(1, -1)))
        U = mx * u + my * v
        up, um = 0.5 * (U + np.abs(U)), 0.5 * (U - np.abs(U))
        rhs -= up[I] * (nt[I] - nt[lo]) + um[I] * (nt[hi] - nt[I])
        lower = -np.where(up[I] > 1e-12, U[lo], 0.0)
        upper = np.where(um[I] < -1e-12, U[hi], 0.0)
        b = b + up[I] - um[I]
        c2 = cb2 / sigma / p.rey * (nul[I] + nt[I])
        side = {}
        for n, to in (("lo", lo), ("hi", hi)):
            met = 0.5 * (mx[I] + mx[to]) * mx[I] + 0.5 * (my[I] + my[to]) * my[I]
            ch = (1.0 + cb2) / sigma / p.rey * 0.5 * (nul[I] + nul[to] + nt[I] + nt[to])
            side[n] = np.maximum(met * (ch - c2), 0.0)
        rhs += side["hi"] * (nt[hi] - nt[I]) - side["lo"] * (nt[I] - nt[lo])
        b = b + side["lo"] + side["hi"]
        bands.append((lower - side["lo"], upper - side["hi"]))
    # source
    ddx = lambda f: 0.5 * (f[1:-1, 2:] - f[1:-1, :-2])  # noqa: E731
    ddy = lambda f: 0.5 * (f[2:, 1:-1] - f[:-2, 1:-1])  # noqa: E731
    vort = np.abs(xy[I] * ddx(u) - xx[I] * ddx(v) + yy[I] * ddy(u) - yx[I] * ddy(v))
    x, y = _grid(a, a.x), _grid(a, a.y)
    xw, yw = a.xv.reshape(p.kmax, p.jmax)[0], a.yv.reshape(p.kmax, p.jmax)[0]
    t1, t2 = p.jtail1 - 1, p.jtail2 - 1                     # first and last wall cell (from 0)
    d = np.hypot(x - xw[t1 - 1], y - yw[t1 - 1])            # off the wall: distance to the trailing edge
    j = np.arange(t1, t2 + 1)
    d[:, j] = np.hypot(x[:, j] - 0.5 * (xw[j - 1] + xw[j]), y[:, j] - 0.5 * (yw[j - 1] + yw[j]))
    n, nu = nt[I], nul[I]
    chi = np.maximum(n / nu, 1e-12)
    fv1 = chi ** 3 / (chi ** 3 + cv1 ** 3)
    fv2 = 1.0 - chi / (1.0 + chi * fv1)
    dfv1 = 3 * cv1 ** 3 * chi ** 2 / nu / (chi ** 3 + cv1 ** 3) ** 2
    dfv2 = (fv2 - 1) / chi / nu + (1 - fv2) ** 2 * (dfv1 + fv1 / chi / nu)
    d2 = np.maximum(d[I] ** 2, 1e-12)
    kd2 = d2 * kap * kap * p.rey
    st = np.maximum(vort + nu / kd2 * chi * fv2, 1e-12)
    r = np.minimum(n / kd2 / st, 10.0)
    g = r + cw2 * (r ** 6 - r)
    sixth = ((1 + cw3 ** 6) / (g ** 6 + cw3 ** 6)) ** (1.0 / 6.0)
    fw = g * sixth
    dst = nu * (fv2 / nu + chi * dfv2) / kd2
    dr = nu * (1 / nu - chi * dst / st) / st / kd2
    dg = dr * (1 + cw2 * (6 * r ** 5 - 1))
    dfw = sixth * dg * (1 - g ** 6 / (g ** 6 + cw3 ** 6))
    pro, des = cb1 * st, cw1 * fw / d2 / p.rey
    dpro = pro * dst / st * n
    ddes = (cw1 * dfw / d2 / p.rey * nu * chi + des) * n
    rhs += pro * n - des * n * n
    b = b + np.maximum(des * n - pro, 0.0) + np.maximum(ddes - dpro, 0.0)
    # line solves (a first-order time step in this configuration unless timeac is 1)
    ts = tscale[I]
    if p.timeac == 1:
        ts = (1.0 + 0.002 * np.sqrt(J[I])) / (1.0 + np.sqrt(J[I]))
        ts = ts / (1.0 + ts / p.h)
    rhs, b = rhs * ts, 1.0 + b * ts
    (aj, cj), (ak, ck) = ((lo * ts, hi * ts) for lo, hi in bands)
    dn = _np_tridiag(aj, b, cj, rhs) * b
    dn = _np_tridiag(ak.T, b.T, ck.T, dn.T).T
    nt[I] = np.maximum(n + dn, 1e-20)
    _np_turbc(a, q, u, v)
    chi = nt / nul
    return q, rho * nt * chi ** 3 / (chi ** 3 + cv1 ** 3)


def _np_tridiag(a, b, c, r):
    """Tridiagonal solves along the last axis."""
    c, r = c.copy(), r.copy()
    n = b.shape[-1]
    for i in range(n):
        w = 1.0 / (b[:, i] - (a[:, i] * c[:, i - 1] if i else 0.0))
        r[:, i] = (r[:, i] - (a[:, i] * r[:, i - 1] if i else 0.0)) * w
        c[:, i] *= w
    for i in range(n - 2, -1, -1):
        r[:, i] -= c[:, i] * r[:, i + 1]
    return r
