"""A launch, an opt-in or a copy that fails inside a training call comes back as its status: on the CPU,
with a program that links the library and answers its CUDA runtime calls itself (launch_failures.cpp)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_every_failed_launch_of_a_training_call_is_reported(tmp_path):
    from boost_and_broadside_b200 import _capi

    exe = str(tmp_path / "launch_failures")
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "launch_failures.cpp"),
                    _capi.LIB_PATH, f"-Wl,-rpath,{os.path.dirname(_capi.LIB_PATH)}", "-Wl,--unresolved-symbols=ignore-in-shared-libs",
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
