"""Runs whose gradient hangs on the branches that minmod and the solvers take where their
operands differ by rounding only (the feet of the waves of a shock tube, states at rest beside
walls, a uniform start), for tests/test_gpu_gradient_branches.py.  The inputs take no
transcendental function, so they are the same on every host.  ``python gradient_cases.py`` on a
machine with a GPU writes tests/golden/gradient_branches.json; the committed file was recorded
before the default build took the forms of pip_fp64_forms.cuh (commit c441562)."""
import json
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
GOLDEN = os.path.join(HERE, "golden", "gradient_branches.json")
sys.path.insert(0, os.path.dirname(HERE))

# name: (kind, nx, ny, steps, alpha_c, seed)
CASES = {
    "tube-64": ("tube", 64, 1, 60, 10.0, 1),
    "tube-301": ("tube", 301, 1, 120, 100.0, 2),
    "tube-1024": ("tube", 1024, 1, 150, 1000.0, 3),
    "tube-10007": ("tube", 10007, 1, 40, 100.0, 4),
    "walls-26x18": ("walls", 26, 18, 30, 100.0, 5),
    "walls-45x97": ("walls", 45, 97, 25, 10.0, 6),
    "walls-139x143": ("walls", 139, 143, 30, 100.0, 7),
    "waves-40x24": ("waves", 40, 24, 50, 10.0, 8),
    "waves-159x111": ("waves", 159, 111, 30, 10.0, 9),
    "waves-512x256-a": ("waves", 512, 256, 50, 10.0, 25),
    "waves-512x256-b": ("waves", 512, 256, 50, 10.0, 38),
    "waves-512x256-c": ("waves", 512, 256, 50, 10.0, 40),
    "waves-512x256-d": ("waves", 512, 256, 50, 10.0, 43),
}


def _unit(rng, shape=None):
    """Multiples of 2^-20 in [0, 1)."""
    return rng.integers(0, 1 << 20, size=shape) / float(1 << 20)


def _field(rng, x, y, kmax):
    """A smooth periodic field on the unit box: integer wave vectors of a quartic wave."""
    f = np.zeros((y.size, x.size))
    for kx in range(-kmax, kmax + 1):
        for ky in range(0, kmax + 1):
            if (kx == 0 and ky == 0) or kx * kx + ky * ky > kmax * kmax:
                continue
            t = kx * x[None, :] + ky * y[:, None] + _unit(rng)
            t = t - np.floor(t)
            u = t * (1.0 - t)
            f = f + (_unit(rng) - 0.5) * (16.0 * (u * u) - 8.0 / 15.0)
    return f / np.max(np.abs(f))


def build(name):
    """(settings, state as a (13, jx, ix) array, cotangent, projections) of a case."""
    from pip_b200 import ics
    from pip_b200.params import Settings
    kind, nx, ny, steps, col, seed = CASES[name]
    rng = np.random.default_rng(seed)
    f_n, f_p, f_p_n, f_p_p = ics.fractions(0.5)
    if kind == "tube":
        s = Settings(ndim=1, ix0=nx, start=(-0.5, -1.0, -1.0), end=(0.5, 1.0, 1.0), n_fraction=0.5,
                     col=col)
        left = (s.coordinates()[0] < 0.1 * (_unit(rng) - 0.5))[None, :]
        ro = np.where(left, 1.0, 1.0 / (4.0 + 6.0 * _unit(rng)))
        pr = np.where(left, 1.0, 1.0 / (5.0 + 10.0 * _unit(rng)))
        by = np.where(left, 1.0, -1.0)
        zero = np.zeros_like(ro)
        vx = vy = bz = zero
        bx = zero + 0.75
    else:
        s = Settings(ndim=2, ix0=nx, jx0=ny, end=(1.0, ny / nx, 1.0), n_fraction=0.5, col=col,
                     flag_bnd=[1] * 6 if kind == "waves" else [10, 10, 2, 2, 1, 1])
        x, y = s.coordinates()[:2]
        y = y * (nx / ny)
        one, zero = np.ones((y.size, x.size)), np.zeros((y.size, x.size))
        ro, pr, bx, by, bz = one, 0.6 * one, one, zero, zero
        vx, vy = 2.0e-2 * _field(rng, x, y, 4), 2.0e-2 * _field(rng, x, y, 4)
        if kind == "walls":
            # at rest and without field at the edges of the box
            w = ((np.maximum(4.0 * x * (1.0 - x), 0.0))[None, :] *
                 (np.maximum(4.0 * y * (1.0 - y), 0.0))[:, None])
            vx, vy = 20.0 * w * vx, 20.0 * w * vy
            bx, by = 0.4 * w * _field(rng, x, y, 3), 0.4 * w * _field(rng, x, y, 3)
    Uh = ics.pv2cq_hd(s, f_n * ro, vx, vy, zero, f_p_n * pr)
    Um = ics.pv2cq_mhd(s, f_p * ro, vx, vy, zero, f_p_p * pr, bx, by, bz)
    U0 = np.concatenate([Um, Uh])
    g = 2.0 * _unit(rng, U0.shape) - 1.0
    return s, U0, g, steps


def measures(name):
    """The gradient of a case as its norm, its largest entry, the derivative along alpha_c and
    eight projections on random fields, each relative to the norms of both."""
    import torch
    from pip_b200.adjoint import AdjointRun, pip_run
    s, U0, g, steps = build(name)
    run = AdjointRun(s, steps, checkpoint_every=25)
    U = torch.from_numpy(U0).cuda().requires_grad_(True)
    col = torch.tensor(s.col, dtype=torch.float64, requires_grad=True)
    UN = pip_run(U, col, run)
    g0, gc = torch.autograd.grad(UN, (U, col), torch.from_numpy(g).cuda())
    run.close()
    G = g0.cpu().numpy()
    norm = float(np.linalg.norm(G))
    rng = np.random.default_rng(99)
    out = {"norm": norm, "max": float(np.abs(G).max()), "col": float(gc), "along": []}
    for _ in range(8):
        w = 2.0 * _unit(rng, G.shape) - 1.0
        out["along"].append(float((w * G).sum() / (np.linalg.norm(w) * norm)))
    return out


if __name__ == "__main__":
    if len(sys.argv) > 2:
        from pip_b200 import capi
        capi.LIB_PATH = os.path.abspath(sys.argv[2])
    with open(sys.argv[1] if len(sys.argv) > 1 else GOLDEN, "w") as fh:
        json.dump({n: measures(n) for n in CASES}, fh, indent=1)
