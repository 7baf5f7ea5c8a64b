"""The tile rows of a split stage (pip_b200/csrc/pip_rows.cuh), compiled for the host: the launch
that the halo exchange waits for holds every row of cells that it sends, at every grid height."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_sent_rows_are_in_the_first_launch(tmp_path):
    exe = tmp_path / "rows_check"
    subprocess.run(["g++", "-O1", "-std=c++17", os.path.join(HERE, "rows_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    assert r.stdout.split() == ["grids", "1782", "wrong", "0"]
