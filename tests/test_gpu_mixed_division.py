"""The mixed form's shared-reciprocal quotients (pip_mixed_cell.cuh) against the IEEE division:
2^30 seeded operands, no difference allowed."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu


def test_quotients_round_as_the_division(tmp_path):
    from pip_b200 import build as b
    here = os.path.dirname(os.path.abspath(__file__))
    exe = tmp_path / "div_check"
    subprocess.run([b.nvcc()] + b.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    os.path.join(here, "div_check.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert out.split() == ["differ", "0", "0", "0"]
