"""Numbers that are found once per device (per_device.hpp), without a device."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_device_has_its_own(tmp_path):
    exe = str(tmp_path / "per_device")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", os.path.join(ROOT, "tests", "cpp", "per_device.cpp"),
                    "-I", os.path.join(ROOT, "umappp_b200", "csrc"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0
