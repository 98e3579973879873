"""Builds the native code in-tree: ``python -m forgetting_transformer_b200.build``.

Two shared objects next to this file, both git-ignored:

* ``libfox_b200.so``: every kernel file compiled by ``nvcc`` for sm_100a only (SASS, no PTX); exports the C ABI declared
  in ``include/fox_b200.h``.  nvcc cross-compiles, so no GPU is needed.
* ``_fox_host.<python>-torch<version>.so``: the operators' host side as a Python extension (``g++`` against the installed
  PyTorch's headers), linked to the first.  PyTorch's C++ interface changes from version to version: the name holds what the
  file was built against, so that one built against another PyTorch is not loaded but built anew.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
import tempfile
from concurrent.futures import ThreadPoolExecutor

import torch

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libfox_b200.so")


def host_path(torch_version: str = torch.__version__) -> str:
    python = sysconfig.get_config_var("SOABI") or sys.implementation.cache_tag
    return os.path.join(PKG_DIR, f"_fox_host.{python}-torch{torch_version}.so")


HOST_PATH = host_path()
SOURCES = ["fox_scan.cu", "fox_attn_fwd.cu", "fox_attn_bwd.cu", "fox_attn_bwd_dq.cu", "fox_attn_bwd_kv.cu", "fox_decode.cu", "fox_normgate.cu", "fox_rmsnorm.cu", "fox_shift.cu", "fox_glu.cu", "fox_ce.cu", "fox_block.cu", "fox_step.cu", "fox_noalloc.cu"]
HEADERS = ["fox_common.cuh", "fox_host.h", os.path.join("..", "..", "include", "fox_b200.h")]
HOST_SOURCES = ["host_module.cpp", "host_attention.cpp", "host_block.cpp", "host_gemm.cpp"]
HOST_HEADERS = ["host_common.h", "host_attention.h", "host_block.h", "host_gemm.h", os.path.join("..", "..", "include", "fox_b200.h")]


def _paths(names):
    return [p for p in (os.path.join(CSRC, s) for s in names) if os.path.exists(p)]


def _stale(target, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def is_stale() -> bool:
    return _stale(LIB_PATH, _paths(SOURCES + HEADERS)) or _stale(HOST_PATH, _paths(HOST_SOURCES + HOST_HEADERS))


def _run(cmd, verbose=False):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    if verbose:
        sys.stderr.write(res.stderr)


def _compile_all(sources, compile_cmd, link_cmd, target, libs=(), verbose=False):
    """Each source to an object file of its own, side by side, then one link (to a temporary name that replaces the
    target, so that a process which has the old file mapped keeps it)."""
    with tempfile.TemporaryDirectory(dir=PKG_DIR, prefix=".build_") as tmp:
        objs = [os.path.join(tmp, os.path.basename(s) + ".o") for s in sources]
        with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as pool:
            list(pool.map(lambda so: _run(compile_cmd + ["-c", so[0], "-o", so[1]], verbose), zip(sources, objs)))
        part = os.path.join(tmp, os.path.basename(target))
        _run(link_cmd + ["-shared", "-o", part] + objs + list(libs))
        os.replace(part, target)


def _build_kernels(verbose):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    flags = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC"]
    _compile_all(_paths(SOURCES), flags + (["-Xptxas", "-v"] if verbose else []), flags, LIB_PATH, verbose=verbose)


def _host_libs():
    """What the extension is linked to: PyTorch's own libraries and the kernels.  The CUDA runtime and cuBLASLt are not named:
    they are those libtorch_cuda depends on, wherever and in whatever version the installed PyTorch has them."""
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    return ["-Wl,--no-as-needed", "-L" + lib, "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda",
            "-L" + PKG_DIR, "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + lib]


def _build_host(verbose):
    from torch.utils.cpp_extension import include_paths
    # (not $CXX: the extension has to share the process's libstdc++, which a compiler that only has the static one breaks)
    cxx = os.environ.get("FOX_B200_CXX", "g++")
    inc = include_paths("cuda") + [sysconfig.get_paths()["include"]]
    flags = [cxx, "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + [f for i in inc for f in ("-isystem", i)]
    _compile_all(_paths(HOST_SOURCES), flags, [cxx], HOST_PATH, _host_libs(), verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _stale(LIB_PATH, _paths(SOURCES + HEADERS)):
        _build_kernels(verbose)
    if force or _stale(HOST_PATH, _paths(HOST_SOURCES + HOST_HEADERS)):
        _build_host(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
