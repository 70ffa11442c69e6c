"""CPU check of the FP64 path's quotients, compiled for the host from the CUDA
headers; no GPU."""
from test_host_mixed import _run_check


def test_host_fp64_quotient(tmp_path):
    _run_check(tmp_path, "host_quot_check")
