"""The FP64 forms of the default build (pip_fp64_forms.cuh) on the device."""
import os
import re
import subprocess

import pytest

pytestmark = pytest.mark.gpu


def test_forms_match_the_literal_ones(tmp_path):
    """Fluxes of 786432 seeded faces against pip_physics.cuh's literal forms on the host: the bounds of
    the paired FP32 solvers (170 roundings of the flux scale for nearby, mirrored and weakly
    magnetised faces, 1.7e4 for unrelated ones, whose energy flux cancels) in FP64, times 16
    for the reordered expressions; states at the floors like unrelated ones (their speeds are
    far above the thermal one).  Limited face states bit for bit; the roots within 2 ulps; no
    mass through a mirror wall."""
    from pip_b200 import build as b
    here = os.path.dirname(os.path.abspath(__file__))
    exe = tmp_path / "fp64_forms_check"
    subprocess.run([b.nvcc()] + b.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    os.path.join(here, "fp64_forms_check.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    print(out)
    m = re.search(r"nonfinite (\d+) wall_mass (\d+) slopes (\d+) sqrt_ulp (\d+) rsqrt_ulp (\d+)", out)
    assert m and [int(v) for v in m.groups()[:3]] == [0, 0, 0]
    assert int(m.group(4)) <= 2 and int(m.group(5)) <= 2
    near, far = 16 * 1.0e-5 * 2.0 ** -29, 16 * 1.0e-3 * 2.0 ** -29
    for k, d, c in re.findall(r"kind (\d) hlld (\S+) hllc (\S+)", out):
        bound = far if k in "05" else near
        assert float(d) <= bound and float(c) <= bound, (k, d, c)
