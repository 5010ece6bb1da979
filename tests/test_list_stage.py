"""The places a list builder's lane stores to (list_stage.cuh, compiled for the host): a warp's lanes may store in any
order, so each has to store its own entries and nothing else."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("most_samples", [0, 1, 5, 8, 20])
def test_any_order_of_lanes(tmp_path, most_samples):
    exe = str(tmp_path / "list_stage")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-x", "c++", os.path.join(ROOT, "tests", "cpp", "list_stage.cpp"),
                    "-I", os.path.join(ROOT, "umappp_b200", "csrc"), "-o", exe], check=True)
    r = subprocess.run([exe, str(most_samples)], capture_output=True, text=True)
    assert r.returncode == 0, "%s wrong entries" % r.stdout.strip()
