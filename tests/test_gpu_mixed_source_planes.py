"""The mixed form's FP64 source on 2D layers with ionisation and recombination, plane by plane
against the FP64 form: density, streamwise momentum and field, and energy within the mixed form's
1e-5 relative L1; the cross-stream planes, a 1e-3 perturbation of the flow, within 1e-5 of the
streamwise ones; the planes along z stay zero."""
import numpy as np
import pytest

from helpers import interior
from pip_b200 import capi, ics
from pip_b200.params import PIP_FP64, PIP_MIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("imp", [0, 1])
@pytest.mark.parametrize("shape", [(17, 33), (32, 14), (61, 45)])
def test_layer_planes(gpu_lib, imp, shape):
    s, Uh, Um = ics.kelvin_helmholtz(*shape, flag_pip_imp=imp)
    out = []
    for prec in (PIP_FP64, PIP_MIXED):
        with capi.Context(s.overrides(precision=prec)) as c:
            c.upload(Uh, Um)
            c.prologue()
            st, _, n = c.run(nsteps=6)
            assert st == 0 and n == 6
            out.append([interior(U, s) for U in c.download()])
    for species, (a, b) in enumerate(zip(*out)):
        size = np.abs(a).reshape(a.shape[0], -1).sum(axis=1)
        off = np.abs(b - a).reshape(a.shape[0], -1).sum(axis=1)
        scale = {0: 0, 1: 1, 2: 1, 4: 4}          # my on the scale of mx
        if species == 1:
            scale.update({5: 5, 6: 5})            # by on the scale of bx
        for n, k in scale.items():
            assert size[k] > 0 and off[n] <= 1e-5 * size[k], (species, n, off[n] / size[k])
        for n in {3, 7} & set(range(a.shape[0])):
            assert not b[n].any()
