"""CPU check of how a wave's candidate pairs are numbered (wave_part), compiled
for the host from the CUDA headers; no GPU."""
from test_host_mixed import _run_check


def test_host_wave_parts(tmp_path):
    _run_check(tmp_path, "host_wave_check")
