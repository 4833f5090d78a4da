"""CPU test of the per-device bookkeeping of kernel attributes
(natural_number_gb300/csrc/device_once.h): tests/cpp/device_once_test.cpp,
compiled with g++; and no kernel attribute is set behind a flag of the whole
process."""
import glob
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "natural_number_gb300", "csrc")


def test_once_a_device(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is not installed")
    exe = str(tmp_path / "device_once_test")
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC,
                           os.path.join(ROOT, "tests", "cpp", "device_once_test.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip() == "ok"


def test_kernel_attributes_are_set_for_each_device():
    flags = re.compile(r"static\s+(const\s+cudaError_t|bool|std::atomic<bool>)\s+\w+")
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        assert not flags.search(open(path).read()), path
