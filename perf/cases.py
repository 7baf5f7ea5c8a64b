"""Performance cases of the two-fluid framework: what its users have it do, through its public
entry points, over the range of grids, precisions and physics that its configurations, tests
and benchmark use.

A case is one call sequence of a driver: host arrays in, a number of time steps on the
device, host arrays out (``capi.Context``), the differentiable run on device tensors
(``adjoint.pip_run``) or an ensemble of independent runs (``ensemble.Ensemble``).  Host
arrays are page-locked, as a driver that exchanges them at every output keeps them.

``exact`` restates the same time loop with whole-array torch operations in 64 bits
(main.f90:31-68, Solver_rot.f90, HLL_rot.f90, PIP_rot.f90, HC_rot.f90); states that stay away
from the density and pressure floors, so the floors' rewrites of the conserved state are
left out.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from pip_b200 import adjoint, capi, ensemble, ics
from pip_b200.params import PIP_FP64, PIP_IR_NLEVEL, PIP_IR_POWERLAW, PIP_MIXED, Settings


def listed():
    return [
        # the 1D shock tube of the test suite and of the first benchmark configuration: a
        # grid of a few thread blocks, so launches and latency count
        {"name": "tube-1024", "kind": "tube", "nx": 1024, "steps": 400, "mixed": False},
        # a small 2D vortex (parameter studies, the smoke run): latency again, 2D kernels
        {"name": "vortex-64", "kind": "vortex", "nx": 64, "ny": 64, "steps": 200, "mixed": False},
        # the headline workload in the plain 64-bit form: 1024 x 1024 Orszag-Tang with
        # divergence cleaning between two outputs
        {"name": "vortex-1024", "kind": "vortex", "nx": 1024, "ny": 1024, "steps": 100,
         "mixed": False},
        # the same in the mixed form, the benchmark's headline number
        {"name": "vortex-1024-mixed", "kind": "vortex", "nx": 1024, "ny": 1024, "steps": 100,
         "mixed": True},
        # a ragged grid between reflecting walls and open ends, no cleaning, the exponential
        # collision form that strong coupling needs
        {"name": "walls-517x333", "kind": "walls", "nx": 517, "ny": 333, "steps": 100},
        # resistive reconnection-like run: uniform eta, three ghost layers
        {"name": "resistive-500x300", "kind": "resistive", "nx": 500, "ny": 300, "steps": 100},
        # a driver that keeps its own time loop and calls cfl and run_solver each step, with
        # the collision coefficient from the temperatures
        {"name": "driver-256", "kind": "driver", "nx": 256, "ny": 256, "steps": 100},
        # the shear layer with ionisation/recombination and implicit conduction at its
        # configured size, 64-bit
        {"name": "layer-2048x1024", "kind": "layer", "nx": 2048, "ny": 1024, "steps": 10,
         "mixed": False},
        # the same physics in the mixed form on half the columns
        {"name": "layer-1024x512-mixed", "kind": "layer", "nx": 1024, "ny": 512, "steps": 10,
         "mixed": True},
        # forward run and gradient of the wave-damping inversion (its configured grid)
        {"name": "gradient-512x256", "kind": "gradient", "nx": 512, "ny": 256, "steps": 50},
        # a batch of shock tubes of different lengths and parameters
        {"name": "ensemble-256", "kind": "ensemble", "runs": 256, "nx": 8192, "steps": 400},
        # the vortex with the 6-level hydrogen model
        {"name": "levels-512", "kind": "levels", "nx": 512, "ny": 512, "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "vortex", "vortex", "walls", "resistive", "driver", "layer",
                       "gradient", "ensemble", "levels"])
    if kind == "tube":
        return {"kind": kind, "nx": _log(rng, 128, 8192), "steps": rng.randint(50, 400),
                "mixed": rng.random() < 0.3}
    if kind == "vortex":
        return {"kind": kind, "nx": _log(rng, 32, 1024), "ny": _log(rng, 32, 1024),
                "steps": rng.randint(20, 100), "mixed": rng.random() < 0.5}
    if kind in ("walls", "resistive", "driver"):
        return {"kind": kind, "nx": _log(rng, 32, 700), "ny": _log(rng, 32, 700),
                "steps": rng.randint(20, 100)}
    if kind == "layer":
        return {"kind": kind, "nx": _log(rng, 128, 2048), "ny": _log(rng, 64, 1024),
                "steps": rng.randint(2, 10), "mixed": rng.random() < 0.5}
    if kind == "gradient":
        return {"kind": kind, "nx": _log(rng, 48, 512), "ny": _log(rng, 32, 256),
                "steps": rng.randint(5, 50)}
    if kind == "ensemble":
        return {"kind": kind, "runs": _log(rng, 16, 256), "nx": _log(rng, 512, 8192),
                "steps": rng.randint(50, 400)}
    return {"kind": kind, "nx": _log(rng, 32, 512), "ny": _log(rng, 32, 512),
            "steps": rng.randint(3, 10)}


# ---------------------------------------------------------------------- inputs

_TABLE = []


def _expint_table():
    """The exponential-integral table every run with the 6-level model loads once."""
    if not _TABLE:
        _TABLE.append(capi.colexp_table(100000))
    return _TABLE[0]


def _vortex_fields(s, rng, lx, ly, tapered=False):
    """Orszag-Tang fields with a random place, strength and pressure, tapered to rest at the
    edges of a box that is not periodic; the neutral and ion states and the uniform ion
    pressure and density."""
    f_n, f_p, f_p_n, f_p_p = ics.fractions(s.n_fraction)
    x, y = s.coordinates()[:2]
    px, py = rng.uniform(0.0, 1.0, 2)
    amp, prs = rng.uniform(0.9, 1.1), rng.uniform(0.95, 1.05)
    X = (x / lx + px)[None, :] + 0.0 * y[:, None]
    Y = (y / ly + py)[:, None] + 0.0 * x[None, :]
    one, zero = np.ones_like(X), np.zeros_like(X)
    ro, p = 25.0 / (36.0 * math.pi), prs * 5.0 / (12.0 * math.pi)
    b0 = amp / math.sqrt(4.0 * math.pi)
    vx, vy = -amp * np.sin(2 * math.pi * Y), amp * np.sin(2 * math.pi * X)
    bx, by = -b0 * np.sin(2 * math.pi * Y), b0 * np.sin(4 * math.pi * X)
    if tapered:
        w = np.sin(math.pi * x / lx)[None, :] * np.sin(math.pi * y / ly)[:, None]
        vx, vy, bx, by = 0.7 * w * vx, 0.7 * w * vy, 0.7 * w * bx, 0.7 * w * by
    Uh = ics.pv2cq_hd(s, f_n * ro * one, vx, vy, zero, f_p_n * p * one)
    Um = ics.pv2cq_mhd(s, f_p * ro * one, vx, vy, zero, f_p_p * p * one, bx, by, zero)
    return Uh, Um, f_p_p * p, f_p * ro


def _tube_fields(s, rng):
    f_n, f_p, f_p_n, f_p_p = ics.fractions(s.n_fraction)
    left = (s.coordinates()[0] < rng.uniform(-0.1, 0.1))[None, :]
    ro = np.where(left, 1.0, 1.0 / rng.uniform(4.0, 10.0))
    pr = np.where(left, 1.0, 1.0 / rng.uniform(5.0, 15.0))
    by = np.where(left, 1.0, -1.0) * rng.uniform(0.8, 1.0)
    zero = np.zeros_like(ro)
    Uh = ics.pv2cq_hd(s, f_n * ro, zero, zero, zero, f_p_n * pr)
    Um = ics.pv2cq_mhd(s, f_p * ro, zero, zero, zero, f_p_p * pr, zero + 0.75, by, zero)
    return Uh, Um


def _members(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["runs"] * 10000 + case["nx"])   # the same for every seed
    out = []
    for _ in range(case["runs"]):
        out.append(ics.shock_tube_member(
            nx=int(round(math.exp(sizes.uniform(math.log(256), math.log(case["nx"]))))),
            col=math.exp(rng.uniform(math.log(0.1), math.log(1.0e4))), pratio=rng.uniform(2, 20),
            dratio=rng.uniform(2, 10), ion_frac=rng.uniform(0.05, 0.95)))
    return out


def _start(case, seed):
    """(settings, U_h, U_m, Nexcite or None) of a single run."""
    rng = np.random.default_rng(seed)
    kind, nx, ny = case["kind"], case["nx"], case.get("ny", 1)
    prec = PIP_MIXED if case.get("mixed") else PIP_FP64
    if kind == "tube":
        s = Settings(ndim=1, ix0=nx, start=(-0.5, -1.0, -1.0), end=(0.5, 1.0, 1.0), n_fraction=0.5,
                     col=100.0, precision=prec)
        return (s,) + _tube_fields(s, rng) + (None,)
    box = dict(ndim=2, ix0=nx, jx0=ny, flag_bnd=[1] * 6, start=(0.0, 0.0, 0.0))
    if kind == "layer":
        s = Settings(ndim=2, ix0=nx, jx0=ny, start=(-1.0, -0.5, 0.0), end=(1.0, 0.5, 1.0),
                     flag_bnd=[1, 1, 2, 2, 1, 1], n_fraction=0.5, col=100.0, flag_ir=PIP_IR_POWERLAW,
                     flag_ir_type=1, ir_chi=5.0, flag_heat=1, kapper=0.01, precision=prec)
        f_n, f_p, f_p_n, f_p_p = ics.fractions(0.5)
        te = 0.5 * f_p_p / f_p                  # ionisation balance of the initial state
        s = s.overrides(ir_rec_coef=1.0, ir_ion_coef=f_p / f_n * math.exp(s.ir_chi / te))
        x, y = s.coordinates()[:2]
        Y = y[:, None] + 0.0 * x[None, :]
        one, zero = np.ones_like(Y), np.zeros_like(Y)
        vx = 0.5 * np.tanh(Y / 0.05)
        vy = rng.uniform(-1e-3, 1e-3, Y.shape) * np.exp(-(Y / 0.1) ** 2)
        Uh = ics.pv2cq_hd(s, f_n * one, vx, vy, zero, f_p_n / s.gm * one)
        Um = ics.pv2cq_mhd(s, f_p * one, vx, vy, zero, f_p_p / s.gm * one, 0.1 * one, zero, zero)
        return s, Uh, Um, None
    if kind == "walls":
        s = Settings(n_fraction=0.5, col=2.0e3, flag_pip_imp=1, end=(1.0, ny / nx, 1.0),
                     **dict(box, flag_bnd=[10, 10, 2, 2, 1, 1]))
    elif kind == "resistive":
        s = Settings(n_fraction=0.9, col=1.0e3, flag_divb=1, flag_resi=1, eta_0=1.0e-4,
                     end=(1.0, ny / nx, 1.0), **box)
    elif kind == "driver":
        s = Settings(n_fraction=0.9, col=1.0e3, flag_divb=1, flag_col=3, end=(1.0, ny / nx, 1.0), **box)
    elif kind == "levels":
        s = Settings(n_fraction=0.9, col=1.0e3, flag_divb=1, flag_ir=PIP_IR_NLEVEL, flag_ir_type=1,
                     t_norm=6500.0, n_norm=1.0e17, t_ir=1.0e-3, end=(1.0, ny / nx, 1.0), **box)
    else:
        s = Settings(n_fraction=0.9, col=1.0e3, flag_divb=1, end=(1.0, ny / nx, 1.0), precision=prec,
                     **box)
    Uh, Um, p_m, ro_m = _vortex_fields(s, rng, 1.0, ny / nx, kind == "walls")
    if kind != "levels":
        return s, Uh, Um, None
    f_p_p_ini = 6500.0 / (0.5 * s.gm * p_m / ro_m) / float(np.float32(5.0) / np.float32(3.0))
    s = s.overrides(f_p_ini=1.0, f_p_p_ini=f_p_p_ini)
    return s, Uh, Um, ics.lte_nexcite(s, Uh[0], Um[0], np.full_like(Um[0], p_m))


def _wave(case, seed):
    """Settings, device state, collision coefficient and cotangent of the gradient case."""
    nx, ny = case["nx"], case["ny"]
    s = Settings(ndim=2, ix0=nx, jx0=ny, end=(1.0, ny / nx, 1.0), flag_bnd=[1] * 6, n_fraction=0.5,
                 col=10.0)
    rng = np.random.default_rng(seed)
    x, y = s.coordinates()[:2]
    X, Y = x[None, :] + 0.0 * y[:, None], y[:, None] + 0.0 * x[None, :]
    dv = ics.velocity_modes(X, Y, 1.0, ny / nx, int(rng.integers(1 << 30)), 2.0e-2, 4)
    U0 = adjoint.wave_damping_state(s, torch.from_numpy(dv[0]), torch.from_numpy(dv[1])).cuda()
    g = torch.from_numpy(rng.standard_normal(tuple(U0.shape))).cuda()
    return s, U0, g


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    v = t.numpy()
    v[...] = a
    return v


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        s, U0, g = _wave(case, seed)
        return {"case": case, "runner": adjoint.AdjointRun(s, case["steps"]),
                "U0": U0.requires_grad_(True),
                "col": torch.tensor(s.col, dtype=torch.float64, requires_grad=True), "g": g}
    if kind == "ensemble":
        members = [(s, _pinned(h), _pinned(m)) for s, h, m in _members(case, seed)]
        return {"case": case, "members": members, "batch": ensemble.Ensemble(members)}
    s, Uh, Um, nex = _start(case, seed)
    ctx = capi.Context(s)
    if nex is not None:
        ctx.set_nlevel(_expint_table())
    return {"case": case, "ctx": ctx, "in": (_pinned(Uh), _pinned(Um)), "nex": nex,
            "out": (_pinned(np.zeros_like(Uh)), _pinned(np.zeros_like(Um)))}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gradient":
        UN = adjoint.pip_run(state["U0"], state["col"], state["runner"])
        g0, gc = torch.autograd.grad(UN, (state["U0"], state["col"]), state["g"])
        return {"state": UN.detach(), "grad": g0, "grad_col": gc}
    if kind == "ensemble":
        batch = state["batch"]
        for r, (_, Uh, Um) in enumerate(state["members"]):
            batch.upload(r, Uh, Um)
        batch.run(max_steps=case["steps"])
        got = [batch.member(r)[:2] for r in range(batch.n)]
        return {"U_h": np.concatenate([h.ravel() for h, _ in got]),
                "U_m": np.concatenate([m.ravel() for _, m in got])}
    ctx = state["ctx"]
    ctx.upload(*state["in"])
    if kind == "levels":
        ctx.set_nexcite(state["nex"])
    ctx.prologue()
    if kind == "driver":
        for _ in range(case["steps"]):
            dt, _ = ctx.cfl()
            ctx.run_solver(dt)
        ctx.cfl()
    else:
        ctx.run(nsteps=case["steps"])
    Uh, Um = ctx.download(*state["out"])
    out = {"U_h": Uh, "U_m": Um}
    if kind == "levels":
        out["nexcite"] = ctx.nexcite()
    return out


def work(case):
    """State read and written once a step (and once over the host link); arithmetic of a
    step per cell: two stages, each with the HLLD and HLLC fluxes of its faces (about 650
    operations a face) and about 300 for the source and the update."""
    kind, steps = case["kind"], case["steps"]
    dims = 1 if kind in ("tube", "ensemble") else 2
    planes = 14 if kind in ("vortex", "resistive", "driver", "levels") else 13
    if kind == "ensemble":
        cells = case["runs"] * (case["nx"] - 256) / max(math.log(case["nx"] / 256.0), 1e-9)
    else:
        cells = case["nx"] * case.get("ny", 1)
    size = 4 if case.get("mixed") or kind == "ensemble" else 8
    state = cells * planes * size
    per_cell = 2 * (650 * dims + 300)
    moved = 2.0 * steps * state + 2.0 * cells * planes * 8
    flops = float(steps) * cells * per_cell
    if kind == "layer":        # about 20 iterations, three 9-point products each, 7 vectors
        moved += steps * 20.0 * cells * size * 12
        flops += steps * 20.0 * cells * 75
    if kind == "levels":       # populations and rates; about 60 table lookups a rate update
        moved += steps * 2.0 * cells * (2 * 6 + 36) * 8
        flops += steps * 4.0 * cells * 2000
    if kind == "gradient":     # forward, its recomputation and the reverse sweep
        moved *= 3.0
        flops *= 4.0
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------------- 64-bit restatement

def _sgn(a):
    return torch.copysign(torch.ones_like(a), a)


def _lo(a, b):
    return torch.where(a <= b, a, b)


def _hi(a, b):
    return torch.where(a >= b, a, b)


def _minmod_faces(V):
    """Left and right states of the inner faces along the last axis (Util_rot.f90:59-76)."""
    X, Y = V[..., 2:] - V[..., 1:-1], V[..., 1:-1] - V[..., :-2]
    t = _sgn(X) * Y
    d = torch.where(torch.minimum(X.abs(), t) > 0.0, torch.where(X.abs() <= t, X, Y),
                    torch.zeros_like(X))
    return (V[..., 1:-1] + 0.5 * d)[..., :-1], (V[..., 1:-1] - 0.5 * d)[..., 1:]


def _hllc(l, r, gm):
    """HLL_rot.f90:615-687; states (ro, vn, vt1, vt2, pr)."""
    def side(v):
        u = torch.stack([v[0], v[0] * v[1], v[0] * v[2], v[0] * v[3], v[4] / (gm - 1.0) +
                         0.5 * v[0] * (v[1] * v[1] + v[2] * v[2] + v[3] * v[3])])
        f = torch.stack([u[1], v[4] + u[1] * v[1], u[2] * v[1], u[3] * v[1], (u[4] + v[4]) * v[1]])
        return u, f, torch.sqrt(gm * v[4] / v[0])
    (ul, fl, cl), (ur, fr, cr) = side(l), side(r)
    sl, sr = 1.03 * _lo(l[1] - cl, r[1] - cr), 1.03 * _hi(l[1] + cl, r[1] + cr)
    sm = ((ur[1] * (sr - r[1]) - ul[1] * (sl - l[1]) + l[4] - r[4]) /
          (ur[0] * (sr - r[1]) - ul[0] * (sl - l[1])))
    pm = sm * ul[0] * (sl - l[1]) - ul[1] * (sl - l[1]) + l[4]

    def star(v, u, s):
        d = u[0] * (s - v[1]) / (s - sm)
        return torch.stack([d, d * sm, d * v[2], d * v[3],
                            ((s - v[1]) * u[4] - v[4] * v[1] + pm * sm) / (s - sm)])

    def th(a):
        return torch.where(a >= 5e-11, torch.ones_like(a),
                           torch.where(a > 0.0, 2e10 * a, torch.zeros_like(a)))
    tl, tm, tr = th(sl), th(sm), 1.0 - th(sr)
    return tr * fr + tl * fl + (1.0 - tl - tr) * (tm * (fl + sl * (star(l, ul, sl) - ul)) +
                                                  (1.0 - tm) * (fr + sr * (star(r, ur, sr) - ur)))


def _hlld(l, r, gm):
    """HLL_rot.f90:691-901; states (ro, vn, vt1, vt2, pr, bn, bt1, bt2)."""
    def side(v):
        bb = v[5] * v[5] + v[6] * v[6] + v[7] * v[7]
        pt, vb = v[4] + 0.5 * bb, v[1] * v[5] + v[2] * v[6] + v[3] * v[7]
        e = v[4] / (gm - 1.0) + 0.5 * v[0] * (v[1] * v[1] + v[2] * v[2] + v[3] * v[3]) + 0.5 * bb
        u = torch.stack([v[0], v[0] * v[1], v[0] * v[2], v[0] * v[3], e, v[5], v[6], v[7]])
        f = torch.stack([u[1], u[1] * v[1] + pt - v[5] * v[5], u[1] * v[2] - v[5] * v[6],
                         u[1] * v[3] - v[5] * v[7], (e + pt) * v[1] - vb * v[5],
                         torch.zeros_like(bb), v[1] * v[6] - v[5] * v[2],
                         v[1] * v[7] - v[5] * v[3]])
        a = gm * v[4] + bb
        d = a * a - 4.0 * gm * v[4] * (v[5] * v[5])
        ok = d > 0.0
        root = torch.where(ok, torch.sqrt(torch.where(ok, d, torch.ones_like(d))), torch.zeros_like(d))
        return u, f, pt, vb, torch.sqrt((a + root) / (2.0 * v[0]))
    ul, fl, pl, vbl, cl = side(l)
    ur, fr, pr, vbr, cr = side(r)
    c = _hi(cl, cr)
    sl, sr = _lo(l[1], r[1]) - c, _hi(l[1], r[1]) + c
    uh = (sr * ur - sl * ul - fr + fl) / (sr - sl)
    sm, bn = uh[1] / uh[0], uh[5]
    pt = pl + l[0] * (sl - l[1]) * (sm - l[1])
    dl, dr = l[0] * (sl - l[1]) / (sl - sm), r[0] * (sr - r[1]) / (sr - sm)
    al, ar = bn.abs() / torch.sqrt(dl), bn.abs() / torch.sqrt(dr)

    def energy(v, u, s, p, vb, y, z, by, bz):
        return ((s - v[1]) * u[4] - p * v[1] + pt * sm +
                bn * (vb - sm * bn - y * by - z * bz)) / (s - sm)

    def single(v, u, f, s, d, p, vb):           # HLLC-G, HLL_rot.f90:776-807
        y, z = uh[2] / uh[0], uh[3] / uh[0]
        w = torch.stack([d, d * sm, d * y, d * z, energy(v, u, s, p, vb, y, z, uh[6], uh[7]),
                         bn, uh[6], uh[7]])
        return s * (w - u) + f

    def star(v, u, s, d, p, vb):                # HLL_rot.f90:813-843
        q = v[0] * (s - v[1]) * (s - sm) - bn * bn
        q = 1.0 / torch.where(q == 0.0, torch.ones_like(q), q)      # zero: HLLC-G is taken
        g = q * (v[0] * (s - v[1]) * (s - v[1]) - bn * bn)
        by, bz = v[6] * g, v[7] * g
        y, z = v[2] - q * bn * v[6] * (sm - v[1]), v[3] - q * bn * v[7] * (sm - v[1])
        return torch.stack([d, d * sm, d * y, d * z, energy(v, u, s, p, vb, y, z, by, bz), bn, by,
                            bz]), y, z
    wl, yl, zl = star(l, ul, sl, dl, pl, vbl)
    wr, yr, zr = star(r, ur, sr, dr, pr, vbr)
    ql, qr, sg = torch.sqrt(dl), torch.sqrt(dr), _sgn(bn)
    k = 1.0 / (ql + qr)
    y2, z2 = (k * (ql * yl + qr * yr + (wr[6] - wl[6]) * sg), k * (ql * zl + qr * zr + (wr[7] - wl[7]) * sg))
    b2 = k * (ql * wr[6] + qr * wl[6] + ql * qr * (yr - yl) * sg)
    c2 = k * (ql * wr[7] + qr * wl[7] + ql * qr * (zr - zl) * sg)
    el = wl[4] - ql * (yl * wl[6] + zl * wl[7] - y2 * b2 - z2 * c2) * sg
    er = wr[4] + qr * (yr * wr[6] + zr * wr[7] - y2 * b2 - z2 * c2) * sg
    s1, s2 = sm - al, sm + ar
    inner_l = torch.stack([dl, dl * sm, dl * y2, dl * z2, el, bn, b2, c2])
    inner_r = torch.stack([dr, dr * sm, dr * y2, dr * z2, er, bn, b2, c2])
    inner = torch.where(sm >= 0.0, s1 * inner_l - (s1 - sl) * wl - sl * ul + fl,
                        s2 * inner_r - (s2 - sr) * wr - sr * ur + fr)
    fan = torch.where(s1 >= 0.0, sl * (wl - ul) + fl, torch.where(s2 <= 0.0, sr * (wr - ur) + fr, inner))
    one = torch.where(sm >= 0.0, single(l, ul, fl, sl, dl, pl, vbl), single(r, ur, fr, sr, dr, pr, vbr))
    fan = torch.where((sl >= sm - 1.001 * al) | (sm + 1.001 * ar >= sr), one, fan)
    return torch.where(sl >= 0.0, fl, torch.where(sr <= 0.0, fr, fan))


class _Exact:
    """The time loop on whole arrays (planes, rows, columns), ghost cells included.  With
    `lengths` the rows are independent 1D runs of these lengths, each with its own dt."""

    def __init__(self, s, rows=None, lengths=None):
        self.s, self.m, self.nvm = s, s.margin[0], s.nvar_m
        self.ndim, self.gm = s.ndim, s.gm
        self.batch = lengths is not None
        dev = dict(device="cuda", dtype=torch.float64)
        self.alpha = None
        ix, jx, _ = s.shape
        m = self.m
        if self.batch:
            self.col = torch.tensor([t.col for t in rows], **dev)[:, None]
            self.dx = torch.tensor([t.coordinates()[3][0] for t in rows], **dev)[:, None]
            n = torch.tensor(lengths, device="cuda")[:, None]
            c = torch.arange(int(max(lengths)) + 2 * m, device="cuda")[None, :] - m
            self.im = torch.minimum(c.clamp(min=0), n - 1)
            self.inside = (c >= 0) & (c < n)
            self.gmin = self.dx.clamp(max=100.0)
            return
        self.col = torch.tensor(s.col, **dev)
        dx, dy = (torch.tensor(v, **dev) for v in s.coordinates()[3:5])
        self.dx = dx[m:-m][None, :] if self.ndim == 2 else dx[m:-m][None, :]
        self.dy = dy[m:-m][:, None] if self.ndim == 2 else None
        self.gmin = (torch.minimum(self.dx, self.dy) if self.ndim == 2 else self.dx).clamp(max=100.0)
        self.im, self.sx = self._images(s.flag_bnd[0:2], ix, 1)
        if self.ndim == 2:
            self.jm, self.sy = self._images(s.flag_bnd[2:4], jx, 2)
        sg = s.safety * float(self.gmin.min())
        self.sg = sg

    def _images(self, codes, n, direction):
        """Interior index and sign of every cell along one axis (Boundary_rot.f90:323-402)."""
        m, k = self.m, n - 2 * self.m
        im, sign = [], np.ones((self.nvm + 5, n))
        for c in range(-m, k + m):
            code = codes[0] if c < 0 else codes[1]
            if 0 <= c < k:
                im.append(c)
            elif code == 1:
                im.append(c % k)
            elif code == 10:
                im.append(min(max(c, 0), k - 1))
            else:
                im.append(-1 - c if c < 0 else 2 * k - 1 - c)
                for q in (direction, 4 + direction, self.nvm + direction):
                    sign[q, c + m] = -1.0
        return torch.tensor(im, device="cuda"), torch.tensor(sign, device="cuda")

    def cells(self, U):
        m = self.m
        return U[..., m:-m, m:-m] if self.ndim == 2 else U[..., m:-m]

    def fill(self, u, signs=True):
        if self.batch:
            return torch.gather(u, 2, self.im.expand(u.shape[0], -1, -1))
        U = u[..., self.im] * (self.sx[: u.shape[0], None, :] if signs else 1.0)
        if self.ndim == 2:
            U = U[..., self.jm, :] * (self.sy[: u.shape[0], :, None] if signs else 1.0)
        return U

    # -- cell functions
    def prim(self, U):
        """Primitives of both species: (ro, vx, vy, vz, pr, b...) and (ro, vx, vy, vz, pr)."""
        n, g = self.nvm, self.gm - 1.0
        k = 0.5 * (U[1] * U[1] + U[2] * U[2] + U[3] * U[3]) / U[0]
        pm = g * (U[4] - k - 0.5 * (U[5] * U[5] + U[6] * U[6] + U[7] * U[7]))
        k = 0.5 * (U[n + 1] ** 2 + U[n + 2] ** 2 + U[n + 3] ** 2) / U[n]
        ph = g * (U[n + 4] - k)
        vm = [U[0], U[1] / U[0], U[2] / U[0], U[3] / U[0], pm] + [U[q] for q in range(5, n)]
        vh = [U[n], U[n + 1] / U[n], U[n + 2] / U[n], U[n + 3] / U[n], ph]
        return torch.stack(vm), torch.stack(vh)

    def coefficient(self, U):
        """alpha_c of a state: constant, or from the temperatures (set_collisional, type 2)."""
        if self.s.flag_col == 1:
            return self.col
        vm, vh = self.prim(U)
        return self.col * torch.sqrt(0.5 * (self.gm * vh[4] / vh[0] + 0.5 * self.gm * vm[4] / vm[0]))

    def rates(self, vm):
        s = self.s
        te = 0.5 * self.gm * vm[4] / vm[0]
        return s.ir_rec_coef / torch.sqrt(te), s.ir_ion_coef / torch.sqrt(te) * torch.exp(-s.ir_chi / te)

    def exchange(self, U, a, dtc):
        """Collisional exchange of source_PIP (PIP_rot.f90:1333-1368)."""
        vm, vh = self.prim(U)
        n, gm = self.nvm, self.gm
        te, nte = 0.5 * gm * vm[4] / vm[0], gm * vh[4] / vh[0]
        w = [U[0] * U[n + q] - U[n] * U[q] for q in (1, 2, 3)]
        dv = [vh[q] - vm[q] for q in (1, 2, 3)]
        if self.s.flag_pip_imp == 0:
            e = a * vh[0] * vm[0] * (0.5 * sum(vh[q] ** 2 - vm[q] ** 2 for q in (1, 2, 3)) +
                                     1.5 / gm * (nte - te))
            return torch.stack([torch.zeros_like(e)] + [a * x for x in w] + [e])
        t = dtc * (U[n] + U[0])
        f = -torch.expm1(-a * t) / t
        nde, de = vh[0], vm[0]
        lam = a * (nde + de)
        kap = 3.0 * (gm - 1.0) * a * (0.5 * nde + de)
        # the ion term multiplies (nvz - vz) by nvz, as PIP_rot.f90:1348 does
        B = -(gm * kap / 3.0 / ((nde + de) * (kap - lam)) *
              (de * (dv[0] * vm[1] + dv[1] * vm[2] + dv[2] * vh[3]) +
               nde * (dv[0] * vh[1] + dv[1] * vh[2] + dv[2] * vh[3])))
        D = -(gm / 6.0 * kap * (de - nde) / ((de + nde) * (kap - 2.0 * lam)) * sum(x * x for x in dv))
        E = torch.exp(-kap * dtc)
        e = -(3.0 / gm * a * de * nde / kap *
              ((E - 1.0) * (nte - te) - (B + D) * E + B * torch.exp(-lam * dtc) +
               D * torch.exp(-2.0 * lam * dtc)) / dtc)
        return torch.stack([torch.zeros_like(e)] + [x * f for x in w] + [e])

    def mass_exchange(self, U, gr, gi):
        vm, vh = self.prim(U)
        a, b = gr * vm[0], gi * vh[0]
        kin = 0.5 * (a * (vm[1] ** 2 + vm[2] ** 2 + vm[3] ** 2) - b * (vh[1] ** 2 + vh[2] ** 2 + vh[3] ** 2))
        return torch.stack([a - b] + [a * vm[q] - b * vh[q] for q in (1, 2, 3)] +
                           [kin - gi * vh[4] / (self.gm - 1.0) + 0.5 * gr * vm[4] / (self.gm - 1.0)])

    # -- fluxes
    def faces(self, vm, vh, cmax):
        """Fluxes through the faces along the last axis; vn and bn in planes 1 and 5."""
        lm, rm = _minmod_faces(vm)
        lh, rh = _minmod_faces(vh)
        fm = _hlld(lm[:8], rm[:8], self.gm)
        if self.nvm == 9:
            fn = 0.5 * (lm[8] + rm[8] - cmax * (rm[5] - lm[5]))
            fp = 0.5 * (cmax * cmax * (lm[5] + rm[5]) - cmax * (rm[8] - lm[8]))
            fm = torch.cat([fm[:5], fn[None], fm[6:8], fp[None]])
        return torch.cat([fm, _hllc(lh, rh, self.gm)])

    def fluxes(self, U, cmax):
        m, n = self.m, self.nvm
        vm, vh = self.prim(U)
        w = slice(m - 2, U.shape[2] - m + 2)
        if self.ndim == 1:
            return self.faces(vm[..., w], vh[..., w], cmax), None
        fx = self.faces(vm[:, m:-m, w], vh[:, m:-m, w], cmax)
        pm = [0, 2, 1, 3, 4, 6, 5, 7] + ([8] if n == 9 else [])
        pa = pm + [n + q for q in (0, 2, 1, 3, 4)]
        h = slice(m - 2, U.shape[1] - m + 2)
        fy = self.faces(vm[pm][:, h, m:-m].transpose(1, 2), vh[[0, 2, 1, 3, 4]][:, h, m:-m].transpose(1, 2),
                        cmax)[pa].transpose(1, 2)
        if self.s.flag_resi:
            fx, fy = fx.clone(), fy.clone()
            self.resistive(U, fx, fy)
        return fx, fy

    def resistive(self, U, fx, fy):
        """resistive_flux with E = eta curl B (Solver_rot.f90:597-636), uniform eta and grid."""
        m, b = self.m, U[5:8]
        dx, dy = 2.0 * float(self.dx[0, 0]), 2.0 * float(self.dy[0, 0])
        c = b[:, 1:-1, 1:-1]
        jx_, jy = (b[2, 2:, 1:-1] - b[2, :-2, 1:-1]) / dy, -(b[2, 1:-1, 2:] - b[2, 1:-1, :-2]) / dx
        jz = (b[1, 1:-1, 2:] - b[1, 1:-1, :-2]) / dx - (b[0, 2:, 1:-1] - b[0, :-2, 1:-1]) / dy
        e = self.s.eta_0 * torch.stack([jx_, jy, jz])
        k = m - 1                                   # the interior starts here in c and e
        x0, x1 = (lambda a: a[:, k:-k, k - 1:-k]), (lambda a: a[:, k:-k, k:a.shape[2] - k + 1])
        es, bs = x0(e) + x1(e), x0(c) + x1(c)
        fx[4] += 0.25 * (es[1] * bs[2] - es[2] * bs[1])
        fx[6] -= 0.5 * es[2]
        fx[7] += 0.5 * es[1]
        y0, y1 = (lambda a: a[:, k - 1:-k, k:-k]), (lambda a: a[:, k:a.shape[1] - k + 1, k:-k])
        es, bs = y0(e) + y1(e), y0(c) + y1(c)
        fy[4] += 0.25 * (es[2] * bs[0] - es[0] * bs[2])
        fy[5] += 0.5 * es[2]
        fy[7] -= 0.5 * es[0]

    # -- one step
    def dt(self, U, extra=None):
        s, gm = self.s, self.gm
        vm, vh = self.prim(self.cells(U))
        cm = torch.sqrt((gm * vm[4] + vm[5] ** 2 + vm[6] ** 2 + vm[7] ** 2) / vm[0])
        # vx^2 + vy^2 + vz^2 of a cell at rest has no gradient
        def speed(v):
            q = v[1] ** 2 + v[2] ** 2 + v[3] ** 2
            return torch.where(q > 0.0, torch.sqrt(torch.where(q > 0.0, q, torch.ones_like(q))),
                               torch.zeros_like(q))
        sg = s.safety * self.gmin
        cand = _lo(sg / (speed(vm) + cm), sg / (speed(vh) + torch.sqrt(gm * vh[4] / vh[0])))
        lim = s.pip_imp_factor if s.flag_pip_imp else min(s.safety, 0.3)
        a = self.col if self.alpha is None else self.alpha
        load = _hi(U[0], U[self.nvm]) * a
        if self.batch:
            w = self.inside[:, self.m:-self.m]
            d = torch.where(w, cand, torch.full_like(cand, 10.0)).amin(1, keepdim=True)
            top = torch.where(self.inside, load, torch.zeros_like(load)).amax(1, keepdim=True)
            return torch.minimum(d, lim / top)
        d = cand.reshape(-1)[torch.argmin(cand)]
        top = load.reshape(-1)[torch.argmax(load)]
        d = torch.where(lim / top < d, lim / top, d)
        if s.flag_ir == PIP_IR_POWERLAW:
            gr, gi = self.rates(self.prim(U)[0])
            d = torch.minimum(d, min(s.safety, 0.1) / torch.maximum(gr, gi).max().clamp(min=1e-5))
        if s.flag_resi:
            d = d.clamp(max=s.safety * float(self.gmin.min()) ** 2 / max(s.eta_0, 1e-8))
        return d if extra is None else torch.minimum(d, extra)

    def stage(self, k, Us, U0, dt, rate):
        """RK stage k (1, 2) from the stage state Us; U0 is changed by the exponential form.
        Returns (updated state, U0)."""
        s, n = self.s, self.nvm
        part = 0.5 * dt if k == 1 else dt
        cmax = self.sg / dt if n == 9 else None
        fx, fy = self.fluxes(Us, cmax)
        u, a0 = self.cells(Us), self.cells(U0)
        if s.flag_col != 1:
            self.alpha = self.coefficient(Us)
        a = self.col if self.alpha is None else self.cells(self.alpha)
        ds = self.exchange(u, a, 0.5 * dt)
        zero = torch.zeros_like(u[5:n])
        if s.flag_pip_imp:
            a0 = a0 + torch.cat([0.5 * dt * ds, zero, -0.5 * dt * ds])
            S = torch.zeros_like(u)
        else:
            S = torch.cat([ds, zero, -ds])
        if rate is not None:
            x = self.mass_exchange(u, *rate)
            S = S + torch.cat([-x, zero, x])
        w = a0 - part / self.dx * (fx[..., 1:] - fx[..., :-1])
        if self.ndim == 2:
            w = w - part / self.dy * (fy[:, 1:, :] - fy[:, :-1, :])
        w = w + part * S
        if n == 9:
            f = math.exp(-(0.5 if k == 1 else 1.0) * s.safety * s.db_clean)
            w = torch.cat([w[:8], f * w[8:9], w[9:]])
        # a0 goes on into the next stage; only its interior is read there
        return self.fill(w), self.fill(a0)

    def step(self, U):
        dt = self.dt(U)
        rate = self.rates(self.prim(self.cells(U))[0]) if self.s.flag_ir == PIP_IR_POWERLAW else None
        U1, U0 = self.stage(1, U, U, dt, rate)
        U2, _ = self.stage(2, U1, U0, dt, rate)
        if self.s.flag_heat:
            U2 = self.conduct(U2, dt)
        return U2

    def run(self, U, steps):
        if self.s.flag_col != 1:
            self.alpha = self.coefficient(U)
        for _ in range(steps):
            U = self.step(U)
        return U

    # -- implicit conduction of the ions (HC_rot.f90:67-140,643-739,468-529)
    def conduct(self, U, dt):
        s, m, gm = self.s, self.m, self.gm
        vm, _ = self.prim(U)
        te = gm * vm[4] / vm[0]
        b = vm[5:8]
        dx, dy = float(self.dx[0, 0]), float(self.dy[0, 0])

        def factors(c0, c1):
            bf = 0.5 * (b[(slice(None),) + c0] + b[(slice(None),) + c1])
            nb = bf / torch.sqrt((bf * bf).sum(0)).clamp(min=1e-5)
            t = 0.5 * (te[c0] + te[c1])
            return nb[0], nb[1], t * t * torch.sqrt(t)
        i, j = slice(m, -m), slice(m, -m)
        ilo, ihi = slice(m - 1, -m - 1), slice(m + 1, U.shape[2] - m + 1)
        jlo, jhi = slice(m - 1, -m - 1), slice(m + 1, U.shape[1] - m + 1)
        eta = s.kapper * dt * (gm - 1.0) / vm[0][j, i] * gm
        xl, xr, yd, yu = (factors(c, (j, i)) for c in ((j, ilo), (j, ihi), (jlo, i), (jhi, i)))
        xx = [-(eta * f[2] * f[0] * f[0] / dx / dx) for f in (xl, xr)]
        yy = [-(eta * f[2] * f[1] * f[1] / dy / dy) for f in (yd, yu)]
        xy = [-(eta / 4.0 / dx / dy * f[0] * f[1] * f[2]) for f in (xl, xr, yd, yu)]
        w = torch.zeros((9,) + eta.shape, dtype=torch.float64, device="cuda")
        w[1], w[2] = xx[0] - (xy[3] - xy[2]), xx[1] + (xy[3] - xy[2])
        w[3], w[4] = yy[0] - (xy[1] - xy[0]), yy[1] + (xy[1] - xy[0])
        w[5], w[6], w[7], w[8] = xy[0] + xy[2], -(xy[1] + xy[2]), -(xy[0] + xy[3]), xy[1] + xy[3]
        w[0] = 1.0 - (w[1] + w[2] + w[3] + w[4])
        for edge, pairs in (((slice(None), 0), ((0, 1), (3, 5), (4, 7))),
                            ((slice(None), -1), ((0, 2), (3, 6), (4, 8))),
                            ((0, slice(None)), ((0, 3), (1, 5), (2, 6))),
                            ((-1, slice(None)), ((0, 4), (1, 7), (2, 8)))):
            for to, frm in pairs:
                w[to][edge] += w[frm][edge]
                w[frm][edge] = 0.0
        pad = torch.nn.functional.pad

        def apply(v):
            q = pad(v, (1, 1, 1, 1))
            c = q[1:-1, 1:-1]
            return (w[0] * c + w[1] * q[1:-1, :-2] + w[2] * q[1:-1, 2:] + w[3] * q[:-2, 1:-1] +
                    w[4] * q[2:, 1:-1] + w[5] * q[:-2, :-2] + w[6] * q[:-2, 2:] + w[7] * q[2:, :-2] +
                    w[8] * q[2:, 2:])
        src = te[j, i]
        x = src.clone()
        r = src - apply(x)
        r0, p = r.clone(), r.clone()
        norm = (src * src).sum()
        for _ in range(300):                         # well below the solver's own target
            if float((r * r).sum() / norm) < 1e-27:
                break
            ap = apply(p)
            rr = (r * r0).sum()
            al = rr / (r0 * ap).sum()
            t = r - al * ap
            at = apply(t)
            om = (t * at).sum() / (at * at).sum()
            x = x + al * p + om * t
            r = src - apply(x)
            p = r + (r * r0).sum() / rr * al / om * (p - om * ap)
        V = U.clone()
        V[4, m:-m, m:-m] += (x - src) * vm[0][j, i] / gm / (gm - 1.0)
        return self.fill(self.cells(V))


class _Levels(_Exact):
    """set_IR type 4: the 6-level hydrogen atom (PIP_rot.f90:232-616,1026-1159)."""

    def __init__(self, s, table):
        super().__init__(s)
        self.tab = torch.from_numpy(table).cuda()

    def interp(self, z):
        """Rows' three-point interpolation of E_0, E_1, E_2 (ionexpfitinterp2)."""
        t = self.tab
        n = t.shape[0]
        lo, hi = t[0, 0], t[-1, 0]
        i = torch.floor((z - lo) / (hi - lo) * float(n)).clamp(1, n - 2).long()
        a, b, c = t[i - 1], t[i], t[i + 1]
        x0, x1, x2 = a[..., 0], b[..., 0], c[..., 0]
        w = [(z - x1) * (z - x2) / ((x0 - x1) * (x0 - x2)), (z - x0) * (z - x2) / ((x1 - x0) * (x1 - x2)),
             (z - x0) * (z - x1) / ((x2 - x0) * (x2 - x1))]
        return [w[0] * a[..., q] + w[1] * b[..., q] + w[2] * c[..., q] for q in (1, 2, 3)]

    def colrat(self, te, ne):
        f32 = lambda v: float(np.float32(v))  # noqa: E731  default-real literals of the Fortran
        kb, me, a0 = f32(1.38064852e-23), f32(9.10938356e-31), f32(5.29e-11)
        gw = [2.0, 8.0, 18.0, 32.0, 50.0, 1.0]
        ei = [v / 13.6 * f32(2.18e-18) for v in (13.6, 3.4, 1.51, 0.85, 0.54, 0.0)]
        rn = [0.45] + [1.94 * k ** -1.57 for k in range(2, 7)]
        bn = [-0.603] + [(4.0 - 18.63 / k + 36.24 / k ** 2 - 28.09 / k ** 3) / k for k in range(2, 7)]
        s = ne * torch.sqrt(8.0 * kb * te / math.pi / me) * 2.0 * math.pi * a0 * a0
        base = 32.0 / 3.0 / math.sqrt(3.0) / math.pi
        cr = [[torch.zeros_like(te) for _ in range(6)] for _ in range(6)]
        for a in range(5):
            i = a + 1.0
            if a == 0:
                g = (1.1330, -0.4059, 0.07014)
            elif a == 1:
                g = (1.0785, -0.2319, 0.02947)
            else:
                g = (0.9935 + 0.2328 / i - 0.1296 / i ** 2, -(0.6282 - 0.5598 / i + 0.5299 / i ** 2) / i,
                     (0.3887 - 1.181 / i + 1.470 / i ** 2) / i ** 2)
            for b in range(a + 1, 5):
                j = b + 1.0
                x = 1.0 - (i / j) ** 2
                fn = base * i / j ** 3 / x ** 3 * (g[0] + g[1] / x + g[2] / x ** 2)
                an = 2.0 * i * i / x * fn
                bb = 4.0 * i ** 4 / j ** 3 / x ** 2 * (1.0 + 4.0 / 3.0 / x + bn[a] / x ** 2)
                y = (ei[a] - ei[b]) / kb / te
                z = rn[a] * x + y
                _, y1, y2 = self.interp(y)
                _, z1, z2 = self.interp(z)
                c = s * i * i / x * y * y * (an * ((1.0 / y + 0.5) * y1 - (1.0 / z + 0.5) * z1) +
                                             (bb - an * math.log(2.0 * i * i / x)) * (y2 / y - z2 / z))
                cr[a][b], cr[b][a] = gw[a] / gw[b] * c, c * torch.exp(-y)
            # the ionisation coefficients, with base*i alone in the first term (PIP_rot.f90:507)
            an = base * i + g[0] / 3.0 + g[1] / 4.0 + g[2] / 5.0
            bb = 2.0 / 3.0 * i * i * (5.0 + bn[a])
            y = ei[a] / kb / te
            z = rn[a] + y
            (y0, y1, y2), (z0, z1, z2) = self.interp(y), self.interp(z)
            c = s * i * i * y * y * (an * (y1 / y - z1 / z) + (bb - an * math.log(2.0 * i * i)) *
                                     (y0 - 2.0 * y1 + y2 - z0 + 2.0 * z1 - z2))
            cr[a][5] = c * torch.exp(y)
        h = 2.0 * math.pi * 9.10938356 * 1.38064852 * te / 6.62607004 / 6.62607004 * f32(1.0e14)
        for a in range(5):
            cr[5][a] = ne * cr[a][5] * gw[a] / 2.0 * h ** -1.5 * torch.exp(ei[a] / kb / te)
        return cr

    def set_ir(self, U):
        s = self.s
        vm, _ = self.prim(U)
        tf = s.t_norm / (float(np.float32(5.0) / np.float32(3.0)) * s.f_p_p_ini / s.f_p_ini)
        self.cr = self.colrat(0.5 * self.gm * vm[4] / vm[0] * s.t_norm / tf, U[0] * s.n_norm / s.n0fac)
        up = sum((self.nex[a] * self.cr[a][5]).clamp(min=0.0) for a in range(5))
        dn = sum((self.nex[5] * self.cr[5][a]).clamp(min=0.0) for a in range(5))
        k = s.t_ir / self.ref
        self.rate = (dn / U[0] * k, up / U[self.nvm] * k)      # recombination, ionisation

    def tendency(self, U, level):
        """Level's sum over the other levels minus its convection by the neutrals."""
        N, n, k = self.nex, self.nvm, self.s.t_ir / self.ref
        d = sum(N[q] * self.cr[q][level] - N[level] * self.cr[level][q] for q in range(6)) * k
        c = torch.zeros_like(d)
        dx, dy = 2.0 * float(self.dx[0, 0]), 2.0 * float(self.dy[0, 0])
        c[:, 1:-1] += (N[level][:, 2:] - N[level][:, :-2])[:, :] / dx * (U[n + 1] / U[n])[:, 1:-1]
        c[1:-1, :] += (N[level][2:] - N[level][:-2]) / dy * (U[n + 2] / U[n])[1:-1]
        return d - c

    def excite(self, U, part):
        new = [(self.nex[q] + part * self.tendency(U, q)).clamp(min=float(np.float32(1e-16)))
               for q in range(5)]
        new[0] = new[0] - (sum(new) - U[self.nvm])
        self.nex = self.fill(self.cells(torch.stack(new + [U[0]])), signs=False)

    def run(self, U, steps, nex):
        s = self.s
        self.nex = nex
        one = torch.full((1, 1), 1.0, dtype=torch.float64, device="cuda")
        ref = self.colrat(one * s.t_norm, one * s.n_norm)
        self.ref = float(sum((nex[5, 0, 0] * ref[5][a]).clamp(min=0.0) for a in range(5)))
        for _ in range(steps):
            self.set_ir(U)
            top = torch.maximum(*self.rate).max().clamp(min=1e-5)
            move = max(float(self.tendency(U, q).max()) for q in range(5))
            dt = self.dt(U, torch.minimum(min(s.safety, 0.1) / top, min(s.safety, 0.01) /
                                          torch.tensor(max(move, 1e-5), device="cuda", dtype=torch.float64)))
            Us = U
            for k in (1, 2):
                self.set_ir(Us)
                new, _ = self.stage(k, Us, U, dt, tuple(self.cells(x) for x in self.rate))
                self.excite(new, 0.5 * dt if k == 1 else dt)
                Us = new
            U = Us
        return U, self.nex


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        s, U0, g = _wave(case, seed)
        U0 = U0.requires_grad_(True)
        col = torch.tensor(s.col, dtype=torch.float64, device="cuda", requires_grad=True)
        e = _Exact(s)

        def one(U, c):
            e.col = c
            return e.step(U)
        U = U0
        for _ in range(case["steps"]):
            U = checkpoint(one, U, col, use_reentrant=False)
        g0, gc = torch.autograd.grad(U, (U0, col), g)
        return {"state": U.detach(), "grad": g0, "grad_col": gc.cpu()}
    if kind == "ensemble":
        members = _members(case, seed)
        n = [s.ix0 for s, _, _ in members]
        ix = max(n) + 4
        U = np.zeros((13, len(n), ix))
        for r, (_, h, m) in enumerate(members):
            U[:8, r, : n[r] + 4], U[8:, r, : n[r] + 4] = m[:, 0], h[:, 0]
            U[:, r, n[r] + 4:] = U[:, r, n[r] + 3: n[r] + 4]
        e = _Exact(members[0][0], [s for s, _, _ in members], n)
        U = e.run(torch.from_numpy(U).cuda(), case["steps"]).cpu()
        return {"U_h": torch.cat([U[8:, r, : n[r] + 4].reshape(-1) for r in range(len(n))]),
                "U_m": torch.cat([U[:8, r, : n[r] + 4].reshape(-1) for r in range(len(n))])}
    s, Uh, Um, nex = _start(case, seed)
    U = torch.from_numpy(np.concatenate([Um, Uh])).cuda()
    out = {}
    with torch.no_grad():
        if kind == "levels":
            e = _Levels(s, _expint_table())
            U = e.fill(e.cells(U))
            U, N = e.run(U, case["steps"], e.fill(e.cells(torch.from_numpy(nex).cuda()), signs=False))
            out["nexcite"] = N
        else:
            e = _Exact(s)
            U = e.run(e.fill(e.cells(U)), case["steps"])
    return dict(out, U_h=U[s.nvar_m:], U_m=U[: s.nvar_m])
