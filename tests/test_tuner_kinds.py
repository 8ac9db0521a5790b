"""The tiling autotuner keeps resident and launched chunks apart (runtime/tuner.cu
on the host): a variant means rows of a warp's tasks in the one and warps of a
CTA's units in the other, so the same buckets have a search and a cache line for
each kind, and cache lines without a kind, of kernels with other row groups, are
not used."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tsunami-hysea_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("kinds") / "kinds_driver")
    cmd = ["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(CUDA, "include"), "-x", "c++",
           os.path.join(CSRC, "runtime", "tuner.cu"), "-x", "c++", os.path.join(ROOT, "tests", "native", "kinds_driver.cpp"),
           "-L" + os.path.join(CUDA, "lib64"), "-lcudart", "-Wl,-rpath," + os.path.join(CUDA, "lib64"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def _run(exe, what, cache=None):
    env = {k: v for k, v in os.environ.items() if k not in ("THY_TILING", "THY_TUNE", "THY_TUNE_CACHE")}
    if cache is not None:
        env["THY_TUNE_CACHE"] = str(cache)
    r = subprocess.run([exe, what], capture_output=True, text=True, env=env, timeout=60)
    assert r.returncode == 0, r.stderr
    return r.stdout.strip().split("\n")


def test_each_kind_has_its_own_search(driver):
    assert _run(driver, "decide") == ["launched done=1 tiling=1,0,2 samples=18", "resident done=1 tiling=0,2,0 samples=18"]


def test_the_cache_file_keeps_the_kinds_apart(driver, tmp_path):
    path = tmp_path / "tune.txt"
    _run(driver, "decide", path)
    assert sorted(line.split()[2:] for line in path.read_text().strip().split("\n")) == [
        ["11", "10", "0", "2", "0"], ["11", "10", "1", "0", "2"]]
    assert _run(driver, "look", path) == ["launched done=1 tiling=1,0,2 samples=0", "resident done=1 tiling=0,2,0 samples=0"]


def test_lines_without_a_kind_are_not_used(driver, tmp_path):
    path = tmp_path / "old.txt"
    path.write_text("unknown 0 11 10 2 2 2\nNVIDIA_B200 148 11 10 2 2 2\n")
    assert _run(driver, "look", path) == ["launched done=0 tiling=0,0,0 samples=0", "resident done=0 tiling=0,0,0 samples=0"]
