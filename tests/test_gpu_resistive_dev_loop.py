"""The device-driven loop (pip_dev_*) with the resistivity recomputed at every stage: its stage 2
forms the next step's dt, cfl_resi's bound among it, where pip_run takes a cfl kernel.  FMA-free
and on one block, times and states are those of pip_run bit for bit, on grids of small tiles
(16, 32 and 64 columns), of large ones and on a ragged one; the bound of every cell of a tile
has to count, so eta is largest in a different row of the tiles each time."""
import numpy as np
import pytest

from pip_b200 import capi, ics

pytestmark = pytest.mark.gpu

LAWS = {"current": dict(flag_resi=22, eta_0=0.03, j_cri=5.5),
        "drift": dict(flag_resi=32, eta_0=2e-2, vd_cri=150.0)}


@pytest.mark.parametrize("shape", [(16, 16), (32, 32), (64, 64), (37, 29), (128, 144)])
@pytest.mark.parametrize("law", sorted(LAWS))
@pytest.mark.parametrize("row", [0, 1, 2, 3])
def test_dev_loop_is_pip_run(gpu_lib, law, shape, row):
    s, Uh, Um = ics.orszag_tang(8, ix0=shape[0], jx0=shape[1], fp_exact=1, **LAWS[law])
    # a sheet of current in the rows of one tile row
    m = s.margin[1]
    Um[5, m + 4 + row] += 0.8
    Um[5, m + 5 + row] -= 0.8
    steps = 6
    with capi.Context(s) as c:
        c.upload(Uh, Um)
        c.prologue()
        want = []
        for _ in range(steps):
            st, t, n = c.run(nsteps=1)
            assert st == 0 and n == 1
            want.append(t)
        h, u = c.download()
    got = []
    with capi.Context(s) as c:
        c.upload(Uh, Um)
        c.prologue()
        c.dev_begin(nsteps=steps)
        for _ in range(steps):
            c.dev_stage(1)
            c.dev_stage(2)
            st, _, t, _ = c.dev_poll()
            assert st == 0
            got.append(t)
        h2, u2 = c.download()
    assert got == want
    np.testing.assert_array_equal(h2, h)
    np.testing.assert_array_equal(u2, u)
