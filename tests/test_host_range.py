"""CPU check of the candidate cells of the mixed kernel's tets against the
reference's range formula, bit for bit, compiled for the host from the CUDA
headers; no GPU."""
from test_host_mixed import _run_check


def test_host_candidate_ranges(tmp_path):
    _run_check(tmp_path, "host_range_check")
