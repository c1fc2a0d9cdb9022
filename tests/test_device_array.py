"""Device arrays after a failed allocation (tests/cpp/device_array_check.cpp): scratch that is kept
while it is large enough must not look large enough when there is no memory behind it."""
import os
import shutil
import subprocess

import pytest

import stormm_b200 as sb
from conftest import ROOT

CUDA = "/usr/local/cuda"


def _run(tmp_path):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include")):
        pytest.skip("no C++ compiler or CUDA headers")
    sb.library()
    exe = str(tmp_path / "device_array_check")
    libdir = os.path.join(ROOT, "stormm_b200")
    cmd = ["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I",
           os.path.join(libdir, "csrc"), "-I", os.path.join(CUDA, "include"),
           os.path.join(ROOT, "tests", "cpp", "device_array_check.cpp"), "-o", exe,
           "-L", libdir, "-lstormm_b200", "-L", os.path.join(CUDA, "lib64"), "-lcudart",
           f"-Wl,-rpath,{libdir}", f"-Wl,-rpath,{os.path.join(CUDA, 'lib64')}"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_failed_allocation_leaves_the_array_empty(tmp_path):
    _run(tmp_path)


@pytest.mark.gpu
def test_failed_allocation_after_a_good_one(tmp_path):
    _run(tmp_path)
