"""Builds ``lib/libeptq_b200.so`` from ``csrc/*.cu`` with nvcc for sm_100a and the host extension
``lib/_eptq_host.*.so`` from ``csrc/host/*.cpp`` with g++, named after the interpreter and the torch it is built for.

Run as ``python -m eptq_b200.build``.  nvcc cross-compiles without a GPU.  The
library has no dependency on torch or Python; it exports the C ABI declared in
``include/eptq_b200.h``.  The host extension links against torch and the library.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB_PATH = LIB_DIR / "libeptq_b200.so"
HEADER = PKG.parent / "include" / "eptq_b200.h"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; the eptq_b200 library cannot be built")
    return cand


def sources():
    return sorted(CSRC.glob("*.cu"))


def _newer(inputs, output: Path) -> bool:
    return not output.exists() or max(p.stat().st_mtime for p in inputs) > output.stat().st_mtime


def needs_build() -> bool:
    return _newer(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [HEADER], LIB_PATH)


def _run(cmd, what: str, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
        print(res.stderr, file=sys.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{res.stdout}\n{res.stderr}")


def build_library(force: bool = False, verbose: bool = False) -> Path:
    """The CUDA library and the host extension, each rebuilt when a source is newer (or always with ``force``).
    The CUDA sources are compiled in parallel and linked once."""
    LIB_DIR.mkdir(exist_ok=True)
    if force or needs_build():
        from concurrent.futures import ThreadPoolExecutor
        from tempfile import TemporaryDirectory
        nvcc = _nvcc()
        with TemporaryDirectory() as tmp:
            objs = [str(Path(tmp) / (src.stem + ".o")) for src in sources()]
            compile_flags = [*NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c"]
            with ThreadPoolExecutor(os.cpu_count() or 1) as pool:
                list(pool.map(lambda so: _run([nvcc, *compile_flags, "-o", so[1], str(so[0])], "nvcc", verbose),
                              zip(sources(), objs)))
            _run([nvcc, *NVCC_FLAGS, "--shared", "-o", str(LIB_PATH), *objs], "nvcc (link)", verbose)
    _build_host(force, verbose)
    return LIB_PATH


def _build_host(force: bool, verbose: bool) -> None:
    from ._lib import host_path
    srcs, path = sorted((CSRC / "host").glob("*.cpp")), host_path()
    if not force and not _newer(srcs + [HEADER], path):
        return
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths
    torch_lib = Path(torch.__file__).resolve().parent / "lib"
    cuda_inc = Path(_nvcc()).resolve().parent.parent / "include"
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-isystem{p}" for p in (*include_paths(), sysconfig.get_paths()["include"], cuda_inc)],
           *map(str, srcs), "-o", str(path), f"-L{torch_lib}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu",
           "-ltorch_python", f"-L{LIB_DIR}", "-l:libeptq_b200.so", "-Wl,-rpath,$ORIGIN"]
    _run(cmd, "g++", verbose)


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
