"""CPU check of a boundary call's sums into the caller's grid in host memory
(adeco_gb300/csrc/host_grid.h), compiled with g++ and, where the compiler has
it, its check for undefined behaviour (misaligned loads); no GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("flags", [[], ["-fsanitize=undefined", "-fno-sanitize-recover=undefined"]], ids=["plain", "ubsan"])
def test_host_grid(tmp_path, flags):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "host_grid_check")
    r = subprocess.run([gxx, "-std=c++17", "-O2", *flags, "-o", exe, os.path.join(HERE, "host_grid_check.cpp")],
                       capture_output=True, text=True)
    if flags and r.returncode != 0 and "ubsan" in r.stderr:
        pytest.skip("no undefined-behaviour sanitizer")
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
