"""CPU check of the cube counts that the FP64 leaf deposit launches with
(MetaGrid::cubes); no GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_host_meta_cubes(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "host_meta_check")
    r = subprocess.run([gxx, "-std=c++17", "-O2", "-o", exe, os.path.join(HERE, "host_meta_check.cpp")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
