"""Split of a row over the blocks of the Okada stage (kernels/kernels.h okada_split)
on the host: every column is covered and no index wraps, up to the widest rows that
an int counts."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tsunami-hysea_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_rows_are_covered(tmp_path):
    exe = str(tmp_path / "okada_split_driver")
    cmd = ["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(CUDA, "include"),
           os.path.join(ROOT, "tests", "native", "okada_split_driver.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    widths = [2, 127, 128, 129, 511, 512, 513, 4096, 1000003, 2**31 - 513, 2**31 - 512, 2**31 - 32, 2**31 - 1]
    cases = [(nx, ny, sms) for nx in widths for ny in (2, 100, 100000) for sms in (1, 148)]
    r = subprocess.run([exe, *(str(v) for c in cases for v in c)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    rows = [tuple(int(v) for v in line.split()) for line in r.stdout.strip().split("\n")]
    assert len(rows) == len(cases) and all(ok == 1 for _, _, ok in rows)
    # the split of ordinary grids: one cell a thread, then four
    of = dict(zip(cases, rows))
    assert of[(512, 100, 148)][:2] == (1, 4) and of[(4096, 100000, 148)][:2] == (4, 8)
