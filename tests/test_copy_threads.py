"""The threads that copy between host arrays and pinned slots (copy_threads.hpp), without a device."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("copy") / "copy_threads")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-pthread", os.path.join(ROOT, "tests", "cpp", "copy_threads.cpp"),
                    "-I", os.path.join(ROOT, "umappp_b200", "csrc"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("helpers", [0, 1, 3])
@pytest.mark.parametrize("first_job", [0, 2 ** 24 - 3])   # the job's number has 24 bits
def test_copies(program, helpers, first_job):
    assert subprocess.run([program, "jobs", str(helpers), str(first_job)], timeout=30).returncode == 0


def test_helpers_sleep_while_a_copy_waits(program):
    """Three helpers that kept asking for work would take 1.5 s of processor time in half a second."""
    r = subprocess.run([program, "idle"], capture_output=True, text=True, timeout=30)
    assert r.returncode == 0 and float(r.stdout) <= 0.15
