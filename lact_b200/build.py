"""Builds the two libraries in-tree: liblact_b200.so (kernels and C ABI; nvcc for sm_100a, cross-compiles without a GPU) and
liblact_b200_torch.so (PyTorch operators on top of it; g++)."""
from __future__ import annotations

import glob
import os
import shutil
import subprocess

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(PKG_DIR, "csrc", "lact_b200.cu")
LIB = os.path.join(PKG_DIR, "liblact_b200.so")
HEADER = os.path.join(os.path.dirname(PKG_DIR), "include", "lact_b200.h")
DEPS = sorted(glob.glob(os.path.join(PKG_DIR, "csrc", "*.cu*"))) + [HEADER]
TORCH_LIB = os.path.join(PKG_DIR, "liblact_b200_torch.so")
TORCH_SRC = sorted(glob.glob(os.path.join(PKG_DIR, "csrc", "native", "*.cpp")))
TORCH_DEPS = sorted(glob.glob(os.path.join(PKG_DIR, "csrc", "native", "*"))) + [HEADER]

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--shared",
              "-Xcompiler", "-fPIC"]


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC")


def is_stale(lib: str = LIB, deps=DEPS) -> bool:
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def torch_stamp() -> str:
    """What the operator library built here carries: it fits the PyTorch it was compiled against and no other."""
    import torch
    return f"lact_b200 operators for PyTorch {torch.__version__};"


def built_for_this_torch(lib: str = TORCH_LIB) -> bool:
    with open(lib, "rb") as f:
        return torch_stamp().encode() in f.read()


def _run(cmd, what: str, verbose: bool) -> None:
    if verbose:
        print(" ".join(cmd))
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(what + " failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)


def build_torch(verbose: bool = False) -> str:
    """Compiles the operator library against the installed PyTorch (the sources in parallel, then one link)."""
    import sysconfig
    import tempfile
    from concurrent.futures import ThreadPoolExecutor

    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(find_nvcc()))
    inc = [f for p in cpp_extension.include_paths() + [os.path.join(cuda, "include"), sysconfig.get_path("include")]
           for f in ("-isystem", p)]
    abi = f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"
    libdir = os.path.join(os.path.dirname(torch.__file__), "lib")
    # the system compiler, as nvcc uses it: its libstdc++ is the shared one PyTorch is linked with (a compiler that links its
    # own statically gives this library a second set of stream facets, and formatting an error message then crashes)
    cxx = shutil.which("g++") or "c++"
    with tempfile.TemporaryDirectory() as tmp:
        objs = [os.path.join(tmp, os.path.basename(s) + ".o") for s in TORCH_SRC]
        stamp = f'-DLACT_TORCH_BUILD="{torch_stamp()}"'
        jobs = [[cxx, "-O2", "-std=c++20", "-fPIC", "-w", abi, stamp, *inc, "-c", s, "-o", o] for s, o in zip(TORCH_SRC, objs)]
        with ThreadPoolExecutor(max(1, min(len(jobs), os.cpu_count() or 1))) as pool:
            list(pool.map(lambda c: _run(c, "g++", verbose), jobs))
        _run([cxx, "-shared", "-o", TORCH_LIB, *objs, "-L" + PKG_DIR, "-l:liblact_b200.so", "-L" + libdir, "-lc10", "-lc10_cuda",
              "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN"], "link", verbose)
    return TORCH_LIB


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles what is missing or older than its sources; returns the path of the kernel library."""
    if force or is_stale():
        cmd = [find_nvcc(), *NVCC_FLAGS, "-o", LIB, SRC]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        _run(cmd, "nvcc", verbose)
    if force or is_stale(TORCH_LIB, TORCH_DEPS) or not built_for_this_torch():
        build_torch(verbose)
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose=True))
