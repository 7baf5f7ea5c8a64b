"""2D grids of an odd number of columns, whose tiles are copied cell by cell (no TMA map
describes such rows): the large tiles with full, partial and single-column last tiles and the
small ones, FMA-free against the oracle bit for bit."""
import pytest

from pip_b200 import ics
from test_gpu_parity import assert_match, run_gpu, run_orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(129, 97), (161, 64), (223, 71), (31, 29)])
def test_bits(nx, ny):
    s, Uh, Um = ics.orszag_tang(8, ix0=nx, jx0=ny, fp_exact=1)
    g = run_gpu(s, Uh, Um, nsteps=4)
    o = run_orc(s, Uh, Um, nsteps=4)
    assert_match(g, o, 0.0, bitwise=True)
