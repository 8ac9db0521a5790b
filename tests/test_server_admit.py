"""Admission of the multi-scenario runtime (runtime/server.cu) on the host, against
stand-ins of the batch and of the CUDA runtime: requests that join together share
the table, the work list and the initial dt, and a failure of these fails the
request that does not fit, not the ones admitted with it."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tsunami-hysea_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
OK, ERR_GPU_MEMORY, ERR_INVALID = 0, 1, 3


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("admit") / "admit_driver")
    cmd = [NVCC, "-x", "cu", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + CSRC,
           "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "native", "admit_driver.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def _statuses(exe, widths):
    r = subprocess.run([exe, *map(str, widths)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    out = {}
    for line in r.stdout.strip().split("\n"):
        rid, status, steps = map(int, line.split())
        assert rid not in out   # each request completes once
        out[rid] = (status, steps)
    return [out[k + 1] for k in range(len(widths))]


@pytest.mark.parametrize("widths", [
    (100, 120, 90),               # nothing fails
    (600,), (100, 600, 120, 90),  # one that does not fit, alone and among others
    (600, 700, 100), (100, 501, 13, 120), (13, 13),
])
def test_a_failure_of_the_common_set_up_fails_one_request(driver, widths):
    for n, (status, steps) in zip(widths, _statuses(driver, widths)):
        want = ERR_GPU_MEMORY if n > 500 else ERR_INVALID if n == 13 else OK
        assert status == want and steps == (4 if want == OK else 0), n
