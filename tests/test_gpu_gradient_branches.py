"""The adjoint's gradient where branches are decided by rounding: a trajectory or a reverse sweep
that rounds otherwise takes other branches and moves single entries by up to a few per cent (shock
tubes) or 1e-3 (uniform starts).  Against the recorded measures of tests/gradient_cases.py; the
same arithmetic gives the same gradient, so only the host's sums may differ: 1e-12 of the norms,
where one entry of the largest case, moved by 1e-3 of the root mean square, moves a projection
by 6e-10."""
import json

import pytest

import gradient_cases as C

pytestmark = pytest.mark.gpu

with open(C.GOLDEN) as fh:
    WANT = json.load(fh)


@pytest.mark.parametrize("name", sorted(C.CASES))
def test_gradient_keeps_its_branches(gpu_lib, name):
    got, want = C.measures(name), WANT[name]
    for k in ("norm", "max", "col"):
        assert abs(got[k] - want[k]) <= 1e-12 * abs(want[k]), (k, got[k], want[k])
    for a, b in zip(got["along"], want["along"]):
        assert abs(a - b) <= 1e-12, (a, b)
