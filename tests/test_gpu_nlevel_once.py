"""The default build's 6-level runs, whose steps take the rates of a state from the cfl that
opens them and form that cfl's terms in the rates kernel, against the oracle, which evaluates
both each time: with the pressure floor acting in every step (the rates are then made again),
in the first steps only, and never; 1D and a ragged 2D grid; a collision rewrite before the
stage's rates.  Tolerance: the drop-in 1e-10 of tests/test_gpu_nlevel.py."""
import pytest

from pip_b200 import ics
from test_gpu_nlevel import check, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pr_lim", [1.0e-8, 0.05, 0.08])
@pytest.mark.parametrize("flag_col", [1, 3])
def test_tube_floors(pr_lim, flag_col):
    s, Uh, Um, nex = ics.nlevel_tube(129, t_ir=0.1, pr_lim=pr_lim, flag_col=flag_col)
    check(run_pair(s, Uh, Um, nex, 12), s)


@pytest.mark.parametrize("shape", [(33, 18), (16, 64)])
@pytest.mark.parametrize("itype", [1, 2])
def test_vortex_ragged(shape, itype):
    s, Uh, Um, nex = ics.nlevel_orszag_tang(16, ix0=shape[0], jx0=shape[1], flag_ir_type=itype,
                                            nlev_deriv=4, t_ir=1.0)
    check(run_pair(s, Uh, Um, nex, 6), s)
