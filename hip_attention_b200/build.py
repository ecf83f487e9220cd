"""Build libhipattn_sm100.so in-tree with nvcc (sm_100a only), and the host extension over it with g++.

    python -m hip_attention_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libhipattn_sm100.so")
HOST = os.path.join(PKG, "_host.so")   # CPython extension: the host path of a call, linked to LIB
SOURCES = ["capi.cu", "scan_stage.cu", "scan_stage_mma.cu", "scan_stage_tcgen05.cu", "scan_query_tiles.cu", "scan_key_tiles.cu", "scan_chunks_strict.cu", "scan_chunks_mma.cu", "select.cu", "bsa_generic.cu", "bsa_mma.cu", "bsa_fp32.cu", "bsa_tcgen05.cu", "bsa_decode.cu", "decode_noalloc.cu", "host_kernels.cu"]
HEADERS = ["common.cuh", "host_kernels.h", "bsa_common.cuh", "scan_common.cuh", "scan_tiles.cuh", "mma_common.cuh", "tcgen05_common.cuh", "rope.cuh", os.path.join("..", "..", "include", "hipattn.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--use_fast_math=false"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    flags = [f for f in NVCC_FLAGS if f != "--use_fast_math=false"]
    if verbose:
        flags += ["-Xptxas", "-v"]
    hdrs = [os.path.join(CSRC, h) for h in HEADERS]
    objs, jobs = [], []
    for s in SOURCES:
        src = os.path.join(CSRC, s)
        obj = os.path.join(CSRC, s[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + hdrs):
            jobs.append([nvcc, *flags, "-c", src, "-o", obj])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stdout + r.stderr

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for out in ex.map(run, jobs):
            if verbose and out:
                print(out)
    if jobs or force or _stale(LIB, objs):
        run([nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"])
    host_src = os.path.join(CSRC, "host.cpp")
    if force or jobs or _stale(HOST, [host_src, os.path.join(CSRC, "host_kernels.h"), hdrs[-1], LIB]):
        import torch
        root = os.path.dirname(torch.__file__)
        cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(nvcc) or nvcc)))
        run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", host_src, "-o", HOST,
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
             *(f"-I{d}" for d in (os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                                  sysconfig.get_paths()["include"], os.path.join(cuda, "include"))),
             f"-L{PKG}", "-l:libhipattn_sm100.so", "-Wl,-rpath,$ORIGIN",
             f"-L{os.path.join(root, 'lib')}", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
