"""The work that a device takes as a resident chunk and the rows of its tasks
(kernels/kernels.h resident_units, resident_rows) on the host, from one SM to the
148 that they were measured on: the search for the rows ends and its tasks fit
the launch, whose blocks hold 512 each."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tsunami-hysea_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("rows") / "rows_driver")
    cmd = ["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(CUDA, "include"),
           os.path.join(ROOT, "tests", "native", "rows_driver.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("sms", [1, 2, 18, 36, 57, 58, 74, 147, 148, 160])
def test_rows_fit_on_every_device(driver, sms):
    r = subprocess.run([driver, str(sms)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    most, broken = (int(v) for v in r.stdout.split())
    assert broken == 0
    assert most == min(3712, 3712 * sms // 148)
