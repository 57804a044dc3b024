"""Build libgca_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU).

    python -m long_context_modeling_b200.build [--force] [--verbose]

The library has no Python or torch dependency: it is a plain C-ABI shared object that the
host layer loads with ctypes.
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libgca_b200.so")
HOST_SOURCE = os.path.join(CSRC, "host_binding.cpp")
HOST_LIB = os.path.join(HERE, "_host.so")              # a Python extension module: tensors in, C ABI calls out

SOURCES = ["api.cu", "gca_simt.cu", "gca_f32_sm100.cu", "gca_csr.cu", "gca_decode.cu", "gca_cache.cu", "lmk_topk.cu", "lmk_tc_sm100.cu", "lmk_grad.cu",
           "gca_fwd_sm100.cu", "gca_bwd_sm100.cu", "gca_bwd_q_sm100.cu", "gca_bwd_kv_sm100.cu", "kv_project_sm100.cu", "skinny_linear.cu", "layer_decode.cu", "win_attn_decode.cu", "vmem.cu"]


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))] + [os.path.join(INCLUDE, "gca_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def _host_stale() -> bool:
    return not os.path.exists(HOST_LIB) or any(os.path.getmtime(d) > os.path.getmtime(HOST_LIB)
                                               for d in (HOST_SOURCE, os.path.join(INCLUDE, "gca_b200.h")))


def _start_host_build() -> subprocess.Popen:
    """The host path is the only part that knows torch; it does not link the library (see its source)."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))), "include")
    include = [INCLUDE, *cpp_extension.include_paths(), sysconfig.get_paths()["include"], cuda]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [a for d in include for a in ("-I", d)] + [HOST_SOURCE, "-o", HOST_LIB, "-L", torch_lib]
    cmd += ["-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda", "-ldl"]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def build(force: bool = False, verbose: bool = False) -> str:
    host = _start_host_build() if force or _host_stale() else None
    try:
        if force or _stale():
            _build_library(force, verbose)
    finally:
        out = host.communicate()[0] if host else ""
    if host and host.returncode != 0:
        raise RuntimeError("the host path did not compile:\n" + out)
    return LIB


def _build_library(force: bool, verbose: bool) -> None:
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    headers = max(os.path.getmtime(d) for d in [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")] +
                  [os.path.join(INCLUDE, "gca_b200.h")])
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(CSRC, src.replace(".cu", ".o"))
        objs.append(obj)
        if not (force or verbose) and os.path.exists(obj) and \
                os.path.getmtime(obj) > max(headers, os.path.getmtime(os.path.join(CSRC, src))):
            continue
        cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
               "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {src}\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.check_call([nvcc, "-shared", "-o", LIB] + objs + ["-lcudart"])


def build_variant(out_dir: str, defines, verbose: bool = False) -> str:
    """Compile the whole library with extra `-D...` flags into `out_dir` (used by the test that
    needs a build whose forward withholds a copy; the in-tree library is not touched)."""
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    os.makedirs(out_dir, exist_ok=True)
    procs, objs = [], []
    for src in SOURCES:
        obj = os.path.join(out_dir, src.replace(".cu", ".o"))
        cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
               "-I", INCLUDE, "-I", CSRC] + list(defines) + ["-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose:
            sys.stderr.write(out)
    lib = os.path.join(out_dir, "libgca_b200_variant.so")
    subprocess.check_call([nvcc, "-shared", "-o", lib] + objs + ["-lcudart"])
    return lib


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
