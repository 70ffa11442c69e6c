"""CPU check of how a wave's candidate pairs are numbered (wave_part, start_bit),
compiled for the host from the CUDA headers with the compiler's check for
undefined behaviour; no GPU."""
import os
import subprocess

import pytest

from adeco_gb300.build import _nvcc
from test_host_mixed import HERE, _run_check


def test_host_wave_parts(tmp_path):
    _run_check(tmp_path, "host_wave_check")


def test_host_wave_parts_no_undefined_behaviour(tmp_path):
    exe = str(tmp_path / "check")
    r = subprocess.run([_nvcc(), "-std=c++17", "-O1", "-Xcompiler", "-fsanitize=undefined,-fno-sanitize-recover=undefined",
                        "-o", exe, os.path.join(HERE, "host_wave_check.cu")], capture_output=True, text=True)
    if r.returncode != 0 and "ubsan" in r.stderr:
        pytest.skip("no undefined-behaviour sanitizer")
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
