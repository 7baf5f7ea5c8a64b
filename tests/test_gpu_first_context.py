"""The first context of a process raises the shared-memory limits of its own stage-kernel instances
only: each extra physics, dimension, tile size and flavour runs in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RUN = """
import ctypes, sys
sys.path.insert(0, %r)
import numpy as np
from pip_b200 import capi, ics
s, Uh, Um = %s
with capi.Context(s) as c:
    c.upload(Uh, Um)
    c.prologue()
    st, t, n = c.run(nsteps=3)
    h, m = c.download()
assert st == 0 and n == 3 and np.isfinite(h).all() and np.isfinite(m).all()
print("ran")
"""
CASES = [
    "ics.brio_wu(64)", "ics.brio_wu(20000)", "ics.brio_wu(20000, flag_pip_imp=1)",
    "ics.brio_wu(64, fp_exact=1)", "ics.orszag_tang(32)", "ics.orszag_tang(160)",
    "ics.orszag_tang(160, flag_col=6)", "ics.orszag_tang(160, flag_resi=1, eta_0=1e-3)",
    "ics.orszag_tang(160, flag_resi=1, eta_0=1e-3, flag_col=3, fp_exact=1)",
    "ics.wave_damping(160, 160)", "ics.kelvin_helmholtz(160, 160, flag_heat=1, kapper=0.1)",
    "ics.kelvin_helmholtz(160, 160)", "ics.orszag_tang(32, flag_resi=1, eta_0=1e-3, flag_col=3)",
]


@pytest.mark.parametrize("case", CASES)
def test_first_context_of_a_process(gpu_lib, case):
    r = subprocess.run([sys.executable, "-c", RUN % (ROOT, case)], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and "ran" in r.stdout, r.stdout + r.stderr
