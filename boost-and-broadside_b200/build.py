"""Build the CUDA shared library of the trunk kernels in-tree with nvcc (sm_100a only).

    python boost-and-broadside_b200/build.py [--force]

The library lands beside this file as ``libbnb_trunk.so``; it is what ``_capi`` loads.  Beside it lands
``_host_path.so``, the CPython module with the host side of a call (csrc/host_path.cpp), linked
against the library.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libbnb_trunk.so")
HOST_MODULE = os.path.join(HERE, "_host_path.so")
SOURCES = ["capi.cu", "exact_kernels.cu", "tensor_kernels.cu", "bullet_kv.cu", "pipelined_tile_kernel.cu", "static_scratch.cu", "grad_kernels.cu", "mlp_kernels.cu", "head_tiles.cu", "policy_tail.cu", "train_attention.cu", "train_mlp.cu", "train_linear.cu", "split_kernels.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the trunk kernels cannot be built")
    return exe


def _stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(HOST_MODULE):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST_MODULE))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", "bnb_trunk.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def _host_compile() -> tuple[str, list[str]]:
    """Object file and compiler command of the host module (torch's own headers and C++ ABI)."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    obj = os.path.join(HERE, "build", "host_path.o")
    os.makedirs(os.path.dirname(obj), exist_ok=True)
    includes = [*cpp_extension.include_paths(), os.path.dirname(os.path.dirname(_nvcc())) + "/include",
                sysconfig.get_paths()["include"], os.path.join(ROOT, "include"), CSRC]
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_API_INCLUDE_EXTENSION_H",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    cmd = ["g++", *flags, *[a for i in includes for a in ("-isystem", i)], "-c", os.path.join(CSRC, "host_path.cpp"), "-o", obj]
    return obj, cmd


def _link_host(obj: str) -> list[str]:
    from torch.utils import cpp_extension

    libs = [a for p in cpp_extension.library_paths() for a in ("-L", p)]
    return ["g++", "-shared", "-o", HOST_MODULE, obj, "-L", HERE, "-l:libbnb_trunk.so", *libs, "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu of csrc/ for sm_100a into one shared library; return its path."""
    if not force and not _stale():
        return LIB
    objs = []
    procs = []
    host_obj, host_cmd = _host_compile()
    procs.append(("host_path.cpp", subprocess.Popen(host_cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src in SOURCES:
        obj = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        os.makedirs(os.path.dirname(obj), exist_ok=True)
        cmd = [_nvcc(), *NVCC_FLAGS, *os.environ.get("BNB_NVCC_FLAGS", "").split(), "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-c",
               os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError(f"nvcc failed on {src}")
    for link in ([_nvcc(), "-shared", "-o", LIB, *objs, "-lcudart"], _link_host(host_obj)):
        r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
