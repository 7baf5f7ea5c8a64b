"""The mixed form's FP64 source (pip_mixed_cell.cuh) against the FP64 form: the explicit and the
exponential exchange, ionisation/recombination, and a density floor that acts (there the momentum
exchange takes the unfloored densities), in 1D and on ragged 2D tiles.  After a few steps the
forms differ by the FP32 rounding of the fluxes: 1e-5 relative L1, the mixed form's bar."""
import numpy as np
import pytest

from helpers import interior, rel_l1
from pip_b200 import capi, ics
from pip_b200.params import PIP_FP64, PIP_MIXED

pytestmark = pytest.mark.gpu


def both(s, Uh, Um, steps):
    out = []
    for prec in (PIP_FP64, PIP_MIXED):
        with capi.Context(s.overrides(precision=prec)) as c:
            c.upload(Uh, Um)
            c.prologue()
            st, _, n = c.run(nsteps=steps)
            assert st == 0 and n == steps
            out.append(c.download())
    return out


@pytest.mark.parametrize("imp,col", [(0, 100.0), (1, 100.0), (1, 1.0e4)])
@pytest.mark.parametrize("ro_lim", [1.0e-8, 0.07])
def test_tube(imp, col, ro_lim):
    s, Uh, Um = ics.brio_wu(129, flag_pip_imp=imp, col=col, ro_lim=ro_lim)
    (ah, am), (bh, bm) = both(s, Uh, Um, 8)
    assert np.isfinite(bh).all() and np.isfinite(bm).all()
    assert rel_l1(interior(bh, s), interior(ah, s)).max() <= 1e-5
    assert rel_l1(interior(bm, s), interior(am, s)).max() <= 1e-5


@pytest.mark.parametrize("imp", [0, 1])
@pytest.mark.parametrize("shape", [(17, 33), (32, 14)])
def test_layer(imp, shape):
    s, Uh, Um = ics.kelvin_helmholtz(*shape, flag_pip_imp=imp)
    (ah, am), (bh, bm) = both(s, Uh, Um, 6)
    for a, b in ((ah, bh), (am, bm)):
        e = rel_l1(interior(b, s), interior(a, s))
        # the y-momenta and By are the 1e-3 perturbation of an O(1) flow
        assert e.max() <= 1e-2 and np.sort(e)[: len(e) // 2].max() <= 1e-5
