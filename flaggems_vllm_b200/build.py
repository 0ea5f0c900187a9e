"""Builds libmoe_sm100.so in-tree with nvcc for sm_100a.

The arch is given as ``-gencode arch=compute_100a,code=sm_100a``: the short
form ``-arch=sm_100a`` makes ptxas reject tcgen05 instructions.
"""

from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmoe_sm100.so")
# CPython extension over torch's C++ API and LIB: the native host path of the operators (csrc/host_ext.cpp)
HOST_EXT = os.path.join(HERE, "_host_ext.so")
STAMP = LIB + ".srchash"
SOURCES = ["common.cu", "grouped_topk.cu", "topk_route.cu", "align.cu", "quant.cu", "gemm_simt.cu", "gemm_tc.cu",
           "gemm_wt.cu", "gemm_w8t.cu", "plan.cu", "route_rows.cu", "layer.cu", "gemm_w8.cu", "gemm_small.cu", "gemm_api.cu", "router_gemm.cu", "ep_pack.cu"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _source_digest() -> str:
    """Hash of every source the library is built from (mtimes do not survive a copy)."""
    h = hashlib.sha256()
    files = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC))
    files.append(os.path.join(os.path.dirname(HERE), "include", "moe_sm100.h"))
    for f in files:
        h.update(os.path.basename(f).encode())
        with open(f, "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()


def needs_build() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(HOST_EXT) or not os.path.exists(STAMP):
        return True
    with open(STAMP) as fh:
        return fh.read().strip() != _source_digest()


def _host_ext_cmd() -> list:
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    return [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
            "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(cuda, "include"),
            os.path.join(CSRC, "host_ext.cpp"), "-o", HOST_EXT, "-L" + HERE, "-l:libmoe_sm100.so",
            "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
            "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every CUDA source into one shared library; returns its path."""
    if not force and not needs_build():
        return LIB
    objs = []
    procs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    for src in SOURCES:
        obj = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
               "-Xcompiler", "-fPIC", "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose and out:
            print(out)
    link = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "--shared", "-o", LIB] + objs
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    r = subprocess.run(_host_ext_cmd(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on host_ext.cpp:\n{r.stdout}")
    with open(STAMP, "w") as fh:
        fh.write(_source_digest())
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose=True))
