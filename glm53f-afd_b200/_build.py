"""Compiles the CUDA sources under csrc/ into libglm53f_kda.so beside this file (nvcc, sm_100a only), and the host module."""
from __future__ import annotations

import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libglm53f_kda.so")
HOST = os.path.join(HERE, "_host.so")  # a Python module: the native host path of the per-layer launches

# The IEEE flags are the reference's (crates/glm53f-kda/build.rs:63-68): the chain, the replays and the prologue
# must not contract a multiply and an add, or a replayed prefix stops matching serial steps bit for bit.
IEEE = ["--fmad=false", "--ftz=false", "--prec-div=true", "--prec-sqrt=true"]
SOURCES = {
    "kda_chain.cu": IEEE,
    "kda_rows.cu": IEEE,
    "kda_conv.cu": IEEE,
    "kda_prefill.cu": IEEE,
    "kda_verify_tc.cu": IEEE,  # the chunked verify: its replay saves must carry the exact path's bits (the same expf)
    "kda_prologue.cu": IEEE,  # the layer prologue in front of the chunked prefill: the chain's prologue arithmetic
    "kda_prefill_sp.cu": [],  # tensor-core prefill: agrees with the chain to rounding, so default FP flags
    "proj_gemm.cu": [],      # the projections: tcgen05 GEMM
    "proj_gemm_pair.cu": [], # the same on SM pairs (cta_group::2) for many rows
    "kda_gather.cu": [],     # host code only: CUDA IPC handles for the full output buffers of a head-sharded prefill
    "fwd_rows.cu": [],       # row gather / scatter and the mark copy: data movement only
}


def nvcc() -> str:
    return os.environ.get("GLM53F_NVCC", "/usr/local/cuda/bin/nvcc")


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers += [os.path.join(INCLUDE, "glm53f_kda.h"), os.path.join(INCLUDE, "glm53f_fwd_rows.h"), os.path.join(INCLUDE, "glm53f_proj.h")]
    objs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    for src, flags in SOURCES.items():
        path = os.path.join(CSRC, src)
        obj = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        if force or _stale(obj, [path] + headers):
            cmd = [nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", *flags,
                   "-I" + CSRC, "-I" + INCLUDE, "-Xcompiler", "-fPIC", "-c", path, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            subprocess.check_call(cmd)
        objs.append(obj)
    if force or _stale(LIB, objs):
        subprocess.check_call([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", LIB, *objs])
    build_host(force)
    return LIB


def host_built_for() -> str:
    """What the host module's binary interface depends on beside its own source."""
    import importlib.metadata
    import sys

    return f"torch {importlib.metadata.version('torch')}, python {sys.version_info.major}.{sys.version_info.minor}"


def _host_stale(src: str) -> bool:
    if _stale(HOST, [src, LIB, os.path.join(INCLUDE, "glm53f_kda.h")]):
        return True
    with open(HOST, "rb") as f:
        return host_built_for().encode() + b"\0" not in f.read()


def build_host(force: bool = False) -> str:
    """csrc/host_calls.cpp against Python's and torch's headers, linked to the library beside it."""
    src = os.path.join(CSRC, "host_calls.cpp")
    if force or _host_stale(src):
        import sysconfig

        import torch

        t = os.path.dirname(torch.__file__)
        cuda = os.path.dirname(os.path.dirname(nvcc()))
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f'-DHOST_BUILT_FOR="{host_built_for()}"', "-I" + INCLUDE,
                               "-I" + sysconfig.get_paths()["include"], "-isystem", os.path.join(t, "include"), "-isystem", os.path.join(cuda, "include"), src,
                               "-o", HOST, "-L" + HERE, "-l:" + os.path.basename(LIB), "-L" + os.path.join(t, "lib"), "-lc10", "-lc10_cuda", "-ltorch_python",
                               "-ltorch_cpu", "-Wl,-rpath,$ORIGIN"])
    return HOST


if __name__ == "__main__":
    print(build(verbose=True))
