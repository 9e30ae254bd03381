"""In-tree build of the CUDA library for sm_100a and of the native call path.

`python -m cachalot_b200.build` (or `build()` from Python) compiles every `csrc/*.cu` with
nvcc into `cachalot_b200/libcachalot_b200.so` (nvcc cross-compiles without a GPU) and
`csrc/host/host.cpp` with the C++ compiler into the extension module `cachalot_b200/_host.so`.
Each is rebuilt only when a source or header is newer than it.  CACHALOT_B200_LIB names another file for the library
(development builds); the extension module is the same for all of them.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from importlib import metadata
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = Path(os.environ.get("CACHALOT_B200_LIB", PKG / "libcachalot_b200.so"))
OBJ_DIR = PKG / "csrc" / "build"
HOST_SRC = CSRC / "host" / "host.cpp"
HOST_LIB = PKG / "_host.so"
HOST_STAMP = OBJ_DIR / "host.stamp"  # what _host.so was compiled for

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC,-O3,-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build cachalot_b200")


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _deps() -> list[Path]:
    return sources() + sorted(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "cachalot_b200.h"]


def needs_build() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    return any(p.stat().st_mtime > t for p in _deps())


def build_host(force: bool = False) -> Path:
    """The extension module that ops.py calls.  It takes the CUDA library's entry points as addresses (_lib.load_host)
    and links torch only; it is built anew for another Python or torch."""
    deps = [HOST_SRC, PKG.parent / "include" / "cachalot_b200.h"]
    made_for = f"python {sys.version}\ntorch {metadata.version('torch')}\n"
    if not force and HOST_LIB.exists() and HOST_STAMP.exists() and HOST_STAMP.read_text() == made_for and \
            all(p.stat().st_mtime <= HOST_LIB.stat().st_mtime for p in deps):
        return HOST_LIB
    from torch.utils import cpp_extension

    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-Wall",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(_torch_cxx11_abi())}", "-I" + sysconfig.get_paths()["include"],
           "-I" + str(Path(_nvcc()).resolve().parents[1] / "include"), *("-isystem" + p for p in cpp_extension.include_paths()),
           str(HOST_SRC), "-o", str(HOST_LIB), *("-L" + p for p in cpp_extension.library_paths()), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu",
           "-lc10_cuda", "-lc10"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"host module failed:\n{res.stdout}\n{res.stderr}")
    OBJ_DIR.mkdir(exist_ok=True)
    HOST_STAMP.write_text(made_for)
    return HOST_LIB


def _torch_cxx11_abi() -> bool:
    import torch

    return torch._C._GLIBCXX_USE_CXX11_ABI


def build(force: bool = False, verbose: bool = False) -> Path:
    if force or needs_build():
        _build_cuda(verbose)
    build_host(force)
    return LIB


def _build_cuda(verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ_DIR.mkdir(exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []
    extra += os.environ.get("CACHALOT_NVCC_EXTRA", "").split()  # development switches (-D...)

    def compile_one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(sources()))) as pool:
        objs = list(pool.map(compile_one, sources()))
    cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-cudart", "static"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
