"""Builds libpolarquant_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m polarquant_kv._build            # from the polarquant-kv_b200 directory

The library lands beside this file so it travels with the source tree; nothing is
installed into site-packages and no JIT cache is used.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys

from polarquant_kv._ext import host_file_name

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(PKG_DIR), "csrc")
INCLUDE = os.path.join(os.path.dirname(os.path.dirname(PKG_DIR)), "include")
LIB_PATH = os.path.join(PKG_DIR, "libpolarquant_b200.so")
HOST_PATH = os.path.join(PKG_DIR, host_file_name())    # native host path of the Python package (CPython extension)
HOST_SOURCE = os.path.join(CSRC, "pq_host.cpp")

SOURCES = ["pq_compress.cu", "pq_dequant.cu", "pq_decode_attn.cu", "pq_prefill_attn.cu", "pq_lse_merge.cu", "pq_qjl.cu",
           "pq_llama_abi.cu", "pq_bridge_attn.cu", "pq_bridge_compress.cu"]
HEADERS = ["pq_common.cuh", "pq_tcgen05.cuh", "pq_bridge.cuh", os.path.join(INCLUDE, "polarquant_b200.h"),
           os.path.join(INCLUDE, "polarquant_llama_abi.h")]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put /usr/local/cuda/bin on PATH")


def _older(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    return any(os.path.getmtime(d) > built for d in deps if os.path.exists(d))


def _stale() -> bool:
    deps = [os.path.join(CSRC, s) for s in SOURCES] + [h if os.path.isabs(h) else os.path.join(CSRC, h) for h in HEADERS]
    return _older(LIB_PATH, deps)


def _start_host_build(force: bool):
    """The compiler process for the host module, or None when it is up to date.  Plain C++ (no device code): torch's headers,
    the C ABI's headers; libraries are found beside the module and in torch's own lib folder."""
    headers = [h for h in HEADERS if os.path.isabs(h)]
    if not force and not _older(HOST_PATH, [HOST_SOURCE] + headers):
        return None
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for inc in cpp_extension.include_paths() + [cuda, sysconfig.get_paths()["include"], INCLUDE]:
        cmd += ["-isystem" if inc != INCLUDE else "-I", inc]
    cmd += [HOST_SOURCE, "-o", HOST_PATH, "-L", PKG_DIR, "-l:libpolarquant_b200.so", "-L", torch_lib, "-lc10", "-lc10_cuda",
            "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-L", os.path.join(os.path.dirname(cuda), "lib64"), "-lcudart",
            "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{torch_lib}"]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish_host_build(proc) -> None:
    if proc is not None:
        out, _ = proc.communicate()
        if proc.returncode != 0:
            raise RuntimeError(f"building the host module failed:\n{out}")


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every kernel for sm_100a, link the shared library and build the host module; returns the library's path."""
    if not force and not _stale():
        _finish_host_build(_start_host_build(False))
        return LIB_PATH
    nvcc = _nvcc()
    objs = []
    build_dir = os.path.join(CSRC, "build")
    os.makedirs(build_dir, exist_ok=True)
    common = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC]
    if verbose:
        common += ["-Xptxas", "-v"]
    common += os.environ.get("PQ_NVCC_FLAGS", "").split()     # extra flags for experiments
    procs = []
    for src in SOURCES:
        path = os.path.join(CSRC, src)
        if not os.path.exists(path):
            continue
        obj = os.path.join(build_dir, src.replace(".cu", ".o"))
        objs.append(obj)
        procs.append((src, subprocess.Popen(common + ["-c", path, "-o", obj], stdout=subprocess.PIPE,
                                            stderr=subprocess.STDOUT, text=True)))
    for src, proc in procs:
        out, _ = proc.communicate()
        if verbose and out:
            print(out)
        if proc.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
    link = [nvcc, "-shared", "-o", LIB_PATH] + objs + ["-lcudart"]
    res = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}")
    _finish_host_build(_start_host_build(force))
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
