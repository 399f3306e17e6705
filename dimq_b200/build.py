"""Build ``libdimq_b200.so`` in-tree with plain ``nvcc`` for sm_100a.

The library is header-light (no torch, no pybind): each ``csrc/*.cu`` compiles in
seconds, and the resulting shared object sits next to this file so that it
travels with the source tree.  ``_host.so`` (``csrc/host.cpp``, plain g++ against the
installed PyTorch's headers) is the Python side's native caller of that library.
"""

from __future__ import annotations

import os
import shutil
import sys
import subprocess
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libdimq_b200.so"
HOST = PKG / "_host.so"
SOURCES = ["pack.cu", "lut_generic.cu", "lut_stream.cu", "lut_mma_stream.cu", "lut_mma_regs.cu", "lut_gemm_tc.cu", "lut_expand_gemm.cu", "aux.cu", "attention.cu", "conv_static.cu", "a4_tc.cu", "c_api.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; dimq_b200 needs the CUDA toolkit to build its sm_100a kernels")


def _stale() -> bool:
    if not LIB.exists() or not HOST.exists():
        return True
    newest = max(p.stat().st_mtime for p in list(CSRC.iterdir()) + [PKG.parent / "include" / "dimq_b200.h"])
    return newest > min(LIB.stat().st_mtime, HOST.stat().st_mtime)


def build(force: bool = False, verbose: bool = False, diag: bool = False) -> Path:
    """Compile every kernel source and link the shared library (no-op when up to date).

    ``diag=True`` builds ``libdimq_b200_diag.so`` instead: the same library with
    ``-DDIMQ_B200_DIAG`` (per-role cycle counters and role-skipping switches of the
    tcgen05 kernel, set through ``dimq_diag_configure``).  Nothing in the package
    loads that file; it is for kernel development.
    """
    if diag:
        return _build(PKG / "libdimq_b200_diag.so", PKG / "build_diag", ["-DDIMQ_B200_DIAG"], verbose)
    if not force and not _stale():
        return LIB
    lib = _build(LIB, PKG / "build", [], verbose)
    _build_host(PKG / "build")
    return lib


def _build_host(objdir: Path) -> None:
    """Compile ``csrc/host.cpp`` against PyTorch and link it to the library beside it."""
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parents[1]
    obj = objdir / "host.cpp.o"
    for cmd in (
        ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden",
         f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
         "-isystem", str(root / "include"), "-isystem", str(root / "include" / "torch" / "csrc" / "api" / "include"),
         "-isystem", str(cuda / "include"), "-isystem", sysconfig.get_paths()["include"],
         "-c", str(CSRC / "host.cpp"), "-o", str(obj)],
        ["g++", "-shared", "-o", str(HOST), str(obj), "-L", str(PKG), "-l:libdimq_b200.so", "-L", str(root / "lib"),
         "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-L", str(cuda / "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN"],
    ):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"building _host.so failed:\n{res.stdout}\n{res.stderr}")


def _build(lib: Path, objdir: Path, extra: list[str], verbose: bool) -> Path:
    nvcc = _nvcc()
    objdir.mkdir(exist_ok=True)

    def compile_one(src: str) -> Path:
        obj = objdir / (src + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            print(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as pool:
        objs = list(pool.map(compile_one, SOURCES))
    cmd = [nvcc, "-shared", "-o", str(lib), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return lib


if __name__ == "__main__":
    print(build(force=True, verbose=bool(os.environ.get("DIMQ_BUILD_VERBOSE")), diag="--diag" in sys.argv))
