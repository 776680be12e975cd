"""Builds libllsa_b200.so (nvcc, sm_100a) and _host.so (g++) in-tree.

    python -m llsa_b200.build [--force] [--verbose]

libllsa_b200.so is a plain C-ABI library (include/llsa_b200.h): it links against
the CUDA runtime only, not against torch or Python.  _host.so is the operators'
host path over it (csrc/host.cpp): dispatcher operators with C++ autograd,
linked against torch.
"""
from __future__ import annotations

import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libllsa_b200.so")
HOST = os.path.join(PKG, "_host.so")
SOURCES = ["capi.cu", "pool.cu", "rope.cu", "front_bwd.cu", "topk.cu", "topk_tc.cu", "transpose.cu", "attn.cu", "attn_generic.cu",
           "attn_fwd_mma.cu", "attn_bwd_mma.cu", "attn_pooled_tc.cu", "attn_pooled_bwd_tc.cu", "attn_pooled_loop_tc.cu", "attn_pooled_bwd_loop_tc.cu", "attn_pooled_dkv_loop_tc.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _host_cmd(obj: str):
    """Compile command of the torch-side host path."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    inc = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    return ["g++", "-O2", "-std=c++20", "-fPIC", "-fvisibility=hidden", "-D_GLIBCXX_USE_CXX11_ABI=%d" % abi, "-DTORCH_API_INCLUDE_EXTENSION_H",
            *["-isystem%s" % i for i in inc], "-c", os.path.join(CSRC, "host.cpp"), "-o", obj]


def _host_link_cmd(obj: str):
    import torch
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "lib64")
    return ["g++", "-shared", "-o", HOST, obj, "-L" + PKG, "-lllsa_b200", "-Wl,-rpath,$ORIGIN", "-L" + lib, "-ltorch", "-ltorch_cpu", "-lc10",
            "-ltorch_cuda", "-lc10_cuda", "-L" + cuda, "-lcudart"]


def _stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(HOST):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(os.path.dirname(PKG), "include", "llsa_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu into one shared library and the host path into another; returns the former's path."""
    if not force and not _stale():
        return LIB
    objdir = os.path.join(PKG, "build")
    os.makedirs(objdir, exist_ok=True)
    procs = []
    for src in SOURCES:
        sp = os.path.join(CSRC, src)
        if not os.path.exists(sp):
            raise FileNotFoundError("listed source %s is missing" % sp)
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", sp, "-o", obj] + (["-Xptxas", "-v"] if verbose else [])
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    host_obj = os.path.join(objdir, "host.o")
    host = subprocess.Popen(_host_cmd(host_obj), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    objs = []
    for src, obj, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError("nvcc failed on %s:\n%s" % (src, out))
        if verbose:
            print(out)
        objs.append(obj)
    cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-lcudart"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout)
    out, _ = host.communicate()
    if host.returncode != 0:
        raise RuntimeError("g++ failed on host.cpp:\n%s" % out)
    r = subprocess.run(_host_link_cmd(host_obj), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("link of the host path failed:\n" + r.stdout)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
