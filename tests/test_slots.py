"""The slots that chain sweeps running at once share (csrc/mfcfd_slots.h),
checked on the host (tests/slot_pool_check.cpp).  Needs g++, no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "3d-mfcfd_b200", "csrc")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("slots") / "slot_pool_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, os.path.join(ROOT, "tests", "slot_pool_check.cpp"),
                    "-o", exe], check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("check", ["leases", "launch_beside_a_run", "threads_share", "block_sizes", "block_size_choice"])
def test_slot_pool(checker, check):
    out = subprocess.run([checker, check], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
