"""CPU checks of the host's meta-cell arithmetic (adeco_gb300/csrc/octree.h): the
cube counts that the FP64 leaf deposit launches with (MetaGrid::cubes) and the
look-ups of zoom requests (MetaIndex); no GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.parametrize("name", ["host_meta_check", "host_near_check"])
def test_host_meta(tmp_path, name):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / name)
    r = subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe, os.path.join(HERE, name + ".cpp"),
                        os.path.join(ROOT, "adeco_gb300", "csrc", "octree.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
