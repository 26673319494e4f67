"""Builds ``libkda_b200.so`` in-tree with nvcc for sm_100a (no JIT cache; the library has a plain C ABI, loaded with
ctypes by hosts of any kind) and ``_host.so``, the native host path of this package over PyTorch's C++ API, with g++."""

from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libkda_b200.so")
SOURCES = ["kda_api.cu", "kda_simt.cu", "kda_simt_state.cu", "kda_aux.cu", "kda_tc.cu", "kda_tc_intra.cu", "kda_bwd_intra.cu", "kda_tc_bwd_wy.cu",
           "kda_decode.cu", "kda_state_seg.cu"]
HOST = os.path.join(PKG, "_host.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--expt-extended-lambda", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False, extra_flags=(), lib_path: str = LIB) -> str:
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(PKG), "include", "kda_b200.h"))
    objdir = os.path.join(PKG, "build" if not extra_flags else "build_" + "_".join(f.strip("-") for f in extra_flags))
    os.makedirs(objdir, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> str:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        path = os.path.join(CSRC, src)
        if force or _stale(obj, [path] + headers):
            cmd = [nvcc, *NVCC_FLAGS, *extra_flags, "-c", path, "-o", obj] + (["-Xptxas", "-v"] if verbose else [])
            r = subprocess.run(cmd, capture_output=True, text=True)
            if verbose:
                sys.stderr.write(r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as ex:
        host = ex.submit(_compile_host, objdir, headers, force) if lib_path == LIB else None
        objs = list(ex.map(compile_one, SOURCES))
    if force or _stale(lib_path, objs):
        r = subprocess.run([nvcc, "-shared", "-o", lib_path, *objs, "-lcudart"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    if host is not None:
        _link_host(host.result(), lib_path, force)
    return lib_path


def _run(cmd, what):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")


def _compile_host(objdir: str, headers, force: bool) -> str:
    src, obj = os.path.join(CSRC, "host.cpp"), os.path.join(objdir, "host.o")
    if force or _stale(obj, [src, headers[-1]]):
        import torch
        from torch.utils import cpp_extension

        inc = [d for p in (*cpp_extension.include_paths(), os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"),
                           sysconfig.get_paths()["include"]) for d in ("-isystem", p)]
        _run(["g++", "-O2", "-fPIC", "-std=c++17", "-DTORCH_API_INCLUDE_EXTENSION_H", "-DTORCH_EXTENSION_NAME=_host",
              f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *inc, "-c", src, "-o", obj], "g++ for host.cpp")
    return obj


def _link_host(obj: str, lib_path: str, force: bool) -> None:
    if force or _stale(HOST, [obj, lib_path]):
        from torch.utils import cpp_extension

        _run(["g++", "-shared", "-o", HOST, obj, f"-L{PKG}", "-l:" + os.path.basename(lib_path),
              *(f"-L{d}" for d in cpp_extension.library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch",
              "-ltorch_python", "-Wl,-rpath,$ORIGIN"], "linking _host.so")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
