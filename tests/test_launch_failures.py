"""A launch, an opt-in or a copy that fails inside a training call comes back as its status: on the CPU,
with a program that links the library and answers its CUDA runtime calls itself (launch_failures.cpp)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from boost_and_broadside_b200 import _capi

    if shutil.which("g++") is None:
        pytest.skip("needs a C++ compiler")
    exe = str(tmp_path_factory.mktemp("launches") / "launch_failures")
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "launch_failures.cpp"),
                    _capi.LIB_PATH, f"-Wl,-rpath,{os.path.dirname(_capi.LIB_PATH)}", "-Wl,--unresolved-symbols=ignore-in-shared-libs",
                    "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("case", range(18))   # six shapes x forward, backward, backward that recomputes
def test_every_failed_launch_of_a_training_call_is_reported(program, case):
    r = subprocess.run([program, str(case)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
