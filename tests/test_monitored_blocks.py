"""lbm_step_monitored's blocks of steps on the CPU (tests/host/monitored_blocks.cpp
with fakes of the launches and copies): every step has a cleared slot and its
result arrives; when a launch fails, the results of the steps queued before it
still arrive, and the call returns the launch's status."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OK, ERR_CUDA, ERR_NOMEM = 0, 2, 3  # lbm_status
NEVER = 1 << 60


@pytest.fixture(scope="module")
def blocks(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("blocks") / "libblocks.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "cudalbm_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host", "monitored_blocks.cpp"), "-o", out], check=True)
    f = ctypes.CDLL(out).monitored_blocks
    u64, p64 = ctypes.c_uint64, ctypes.POINTER(ctypes.c_uint64)
    f.argtypes, f.restype = [u64, u64, u64, u64, p64, p64], ctypes.c_int

    def call(n, block, fail_step=NEVER, fail_copy=NEVER):
        res, counts = np.zeros(max(n, 1), np.uint64), np.zeros(3, np.uint64)
        s = f(n, block, fail_step, fail_copy, res.ctypes.data_as(p64), counts.ctypes.data_as(p64))
        return s, res[:n].astype(int), counts.astype(int).tolist()

    return call


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 27])
def test_every_step_has_its_result(blocks, n):
    s, res, counts = blocks(n, 8)
    assert s == OK and res.tolist() == list(range(1, n + 1))
    assert counts == [n, -(-n // 8), -(-n // 8)]


@pytest.mark.parametrize("at", [0, 1, 5, 7, 8, 9, 15, 16, 19])
def test_a_failed_launch_keeps_the_results_before_it(blocks, at):
    s, res, counts = blocks(20, 8, fail_step=at)
    assert s == ERR_CUDA and counts[0] == at
    assert res.tolist() == list(range(1, at + 1)) + [0] * (20 - at)


def test_a_failed_copy_is_reported_and_does_not_hide_a_failed_launch(blocks):
    s, res, counts = blocks(20, 8, fail_copy=1)
    assert s == ERR_NOMEM and counts == [16, 2, 2]
    assert res.tolist() == list(range(1, 9)) + [0] * 12
    assert blocks(20, 8, fail_step=11, fail_copy=1)[0] == ERR_CUDA
