"""Split stages (pip_dev_stage_split) of grids that take the small tiles: as the whole stages and
pip_run bit for bit, in every FP64 flavour and with each extra physics of the stage kernels."""
import numpy as np
import pytest

from pip_b200 import capi, ics

pytestmark = pytest.mark.gpu

CASES = {
    "vortex": lambda nx, ny: ics.orszag_tang(8, ix0=nx, jx0=ny),
    "vortex-exact": lambda nx, ny: ics.orszag_tang(8, ix0=nx, jx0=ny, fp_exact=1),
    "vortex-col": lambda nx, ny: ics.orszag_tang(8, ix0=nx, jx0=ny, flag_col=6),
    "vortex-eta": lambda nx, ny: ics.orszag_tang(8, ix0=nx, jx0=ny, flag_resi=1, eta_0=2e-3),
    "vortex-eta-col": lambda nx, ny: ics.orszag_tang(8, ix0=nx, jx0=ny, flag_resi=1, eta_0=2e-3,
                                                     flag_col=3),
    "vortex-imp": lambda nx, ny: ics.orszag_tang(8, ix0=nx, jx0=ny, flag_pip_imp=1, col=1.0e3),
    "layer-ir": lambda nx, ny: ics.kelvin_helmholtz(nx, ny),
    "waves": lambda nx, ny: ics.wave_damping(nx, ny, amp=1.0e-2),
}


@pytest.mark.parametrize("shape", [(16, 16), (33, 18), (64, 64), (40, 29)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_split_is_whole(gpu_lib, case, shape):
    s, Uh, Um = CASES[case](*shape)
    steps, out = 8, []
    for how in ("run", "whole", "split"):
        with capi.Context(s) as c:
            c.upload(Uh, Um)
            if how == "run":
                st, t, n = c.run(nsteps=steps)
            else:
                c.dev_begin(nsteps=steps)
                for _ in range(steps):
                    for k in (1, 2):
                        if how == "whole":
                            c.dev_stage(k)
                        else:
                            c.dev_stage_split(k)
                st, _, t, n = c.dev_poll()
            assert st == 0 and n == steps
            out.append((t,) + tuple(c.download()))
    for t, h, m in out[1:]:
        assert t == out[0][0]
        np.testing.assert_array_equal(h, out[0][1])
        np.testing.assert_array_equal(m, out[0][2])
