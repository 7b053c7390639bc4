"""Build recipe of ``libsapa_b200.so`` (nvcc, sm_100a only, no torch headers: seconds per file) and of ``_host.so``, the
native host path (g++ with the torch headers; calls the library through its C ABI).

    python -m sapa_b200.build [--force]

The library is built in-tree next to this file so that it travels with the source tree.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libsapa_b200.so")
SOURCES = ["api.cu", "sapa_b.cu", "sapa_mma.cu", "sapa_tma.cu", "sapa_gath_mma.cu", "sapa_d.cu", "sapa_proj.cu", "sapa_proj_mm.cu",
           "sapa_nhwc.cu"]
HEADERS = [os.path.join(CSRC, "common.cuh"), os.path.join(CSRC, "tma_util.cuh"), os.path.join(CSRC, "umma_util.cuh"), os.path.join(CSRC, "finite.cuh"), os.path.join(CSRC, "sapa_gath_umma.cuh"), os.path.join(CSRC, "sapa_strip.cuh"), os.path.join(CSRC, "sapa_strip_fwd.cuh"), os.path.join(CSRC, "sapa_strip_sim.cuh"), os.path.join(CSRC, "sapa_strip_sim16.cuh"), os.path.join(CSRC, "proj_mm.h"), os.path.join(CSRC, "sapa_wide16.cuh"), os.path.join(CSRC, "sapa_gath_wide16.cuh"),
           os.path.join(INCLUDE, "sapa_b200.h")]

HOST = os.path.join(HERE, "_host.so")
HOST_TAG = os.path.join(HERE, "build", "_host.tag")      # what _host.so was built for
HOST_SOURCES = [os.path.join(CSRC, f) for f in ("host.cpp", "host_sapa.inc", "host_deform.inc", "host_module.inc")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libsapa_b200.so")
    return exe


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in SOURCES] + HEADERS + [os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def host_tag() -> str:
    """What a build of the host path is tied to: this torch, its C++ ABI and this Python."""
    import sysconfig

    import torch

    return f"torch {torch.__version__}, C++11 ABI {int(torch._C._GLIBCXX_USE_CXX11_ABI)}, Python {sysconfig.get_config_var('EXT_SUFFIX')}"


def built_host_tag() -> str | None:
    """``host_tag()`` of the build that is there, None when it is not recorded."""
    try:
        with open(HOST_TAG) as f:
            return f.read()
    except OSError:
        return None


def _build_host() -> None:
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    include = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    libs = cpp_extension.library_paths()
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{p}" for p in include), HOST_SOURCES[0], "-o", HOST,
           *(f"-L{p}" for p in libs), *(f"-Wl,-rpath,{p}" for p in libs), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
           "-ltorch_cuda", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for host.cpp:\n{r.stdout}\n{r.stderr}")
    os.makedirs(os.path.dirname(HOST_TAG), exist_ok=True)
    with open(HOST_TAG, "w") as f:
        f.write(host_tag())


def _host_stale() -> bool:
    deps = HOST_SOURCES + [HEADERS[-1], os.path.abspath(__file__)]
    return not os.path.exists(HOST) or built_host_tag() != host_tag() or any(os.path.getmtime(d) > os.path.getmtime(HOST) for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every CUDA source for sm_100a and link the shared library, and the host path; returns the library's path."""
    with ThreadPoolExecutor(max_workers=1) as ex:
        host = ex.submit(_build_host) if force or _host_stale() else None
        _build_lib(force, verbose)
        if host is not None:
            host.result()
    return LIB


def _build_lib(force: bool, verbose: bool) -> None:
    if not force and not _stale():
        return
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)

    def compile_one(src: str) -> str:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    r = subprocess.run([nvcc, "-shared", "-o", LIB, *objs, "-lcudart"], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
