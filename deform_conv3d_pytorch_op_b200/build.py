"""Build recipe for ``csrc/libdcn.so`` (hand-written CUDA for sm_100a, linked by nvcc, no torch headers) and for
``_dcn_torch.so`` (host side of the autograd Functions: C++ against torch, calls libdcn.so through its C ABI).

Run ``python -m deform_conv3d_pytorch_op_b200.build`` or call :func:`build`.  Both are built
in-tree.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc")
LIB = os.path.join(CSRC, "libdcn.so")
BINDING = os.path.join(os.path.dirname(CSRC), "_dcn_torch.so")
BINDING_SOURCE = os.path.join(CSRC, "dcn_torch.cpp")
SOURCES = ["dcn_api.cu", "dcn_simt.cu", "dcn_exact.cu", "dcn_tc.cu"]
HEADERS = ["dcn_common.cuh", "dcn_internal.h", os.path.join("..", "..", "include", "dcn.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"] + os.environ.get("DCN_NVCC_EXTRA", "").split()


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: libdcn.so cannot be built")
    return exe


def is_stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(BINDING):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(BINDING))
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS]
    deps += [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h", ".cu", ".cpp"))]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _binding_command() -> list:
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
             "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
            + [a for p in ext.include_paths() for a in ("-isystem", p)]
            + ["-isystem", os.path.join(cuda, "include"), "-isystem", sysconfig.get_paths()["include"],
               BINDING_SOURCE, "-o", BINDING, "-L" + CSRC, "-l:libdcn.so", "-L" + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu",
               "-ltorch", "-ltorch_python", "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN/csrc"])


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu of the package into ``csrc/libdcn.so`` and the torch binding over it; returns libdcn's path."""
    if not force and not is_stale():
        return LIB
    nvcc = _nvcc()
    objs = []
    procs = []
    for s in SOURCES:
        obj = os.path.join(CSRC, s.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc] + NVCC_FLAGS + ["-c", os.path.join(CSRC, s), "-o", obj]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for cmd, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode != 0:
            sys.stderr.write(out)
        if pr.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    subprocess.check_call([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs)
    subprocess.check_call(_binding_command())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
