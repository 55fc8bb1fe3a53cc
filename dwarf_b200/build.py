"""Builds libdsqg_b200.so (hand-written sm_100a CUDA behind a C ABI) in-tree with nvcc, and _dsqg_torch.so (the
native host side of the Python operators, linked against it) with g++."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")
LIB_PATH = os.path.join(PKG_DIR, "libdsqg_b200.so")
EXT_PATH = os.path.join(PKG_DIR, "_dsqg_torch.so")
SOURCES = ["dsqg_capi.cu", "dsqg_dispatch.cu", "dsqg_generic.cu", "dsqg_decode.cu", "dsqg_mma.cu", "dsqg_mma_d64.cu", "dsqg_mma_window.cu", "dsqg_mma_widths.cu", "dsqg_staged.cu", "dsqg_umma.cu", "dsqg_static.cu", "dsqg_gate.cu", "dsqg_scan.cu", "dsqg_layer.cu", "dsqg_wgrad.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: libdsqg_b200.so cannot be built")
    return cand


def _torch_flags():
    """Compile and link flags of an extension of the installed torch."""
    import torch
    root = os.path.dirname(torch.__file__)
    inc, lib = os.path.join(root, "include"), os.path.join(root, "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    comp = ["-I", inc, "-I", os.path.join(inc, "torch", "csrc", "api", "include"), "-I", os.path.join(cuda, "include"),
            "-I", sysconfig.get_paths()["include"], "-DTORCH_EXTENSION_NAME=_dsqg_torch",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    return comp, ["-L", lib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-Wl,-rpath,{lib}",
                  "-L", os.path.join(cuda, "lib64"), "-lcublasLt", "-lcublas"]


def _stale() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(EXT_PATH):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(EXT_PATH))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, "dsqg_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ for sm_100a and link libdsqg_b200.so next to this file; compile and link the
    torch extension beside it."""
    if not force and not _stale():
        return LIB_PATH
    nvcc = _nvcc()
    objs = []
    build_dir = os.path.join(PKG_DIR, "build")
    os.makedirs(build_dir, exist_ok=True)
    procs = []
    comp, link_ext = _torch_flags()
    ext_obj = os.path.join(build_dir, "dsqg_torch.o")
    jobs = [("dsqg_torch.cpp", ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-I", INCLUDE, *comp,
                                "-c", os.path.join(CSRC, "dsqg_torch.cpp"), "-o", ext_obj])]
    for src in SOURCES:
        obj = os.path.join(build_dir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas"); cmd.insert(2, "-v")
        jobs.append((src, cmd))
        objs.append(obj)
    for src, cmd in jobs:
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out, file=sys.stderr)
        if p.returncode != 0:
            raise RuntimeError(f"compiling {src} failed:\n{out}")
    subprocess.check_call([nvcc, "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart", "-ldl"])
    subprocess.check_call(["g++", "-shared", "-o", EXT_PATH, ext_obj, "-L", PKG_DIR, "-ldsqg_b200", "-Wl,-rpath,$ORIGIN", *link_ext])
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
