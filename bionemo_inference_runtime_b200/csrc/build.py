"""Builds libb200ta.so (sm_100a only) and the layers' native host path (_host.so) next to the package.

Usage: ``python -m bionemo_inference_runtime_b200.csrc.build [--force] [--verbose]``.
The library is linked against the static CUDA runtime and resolves the one
driver symbol it needs at run time, so it loads on machines without a GPU.
"""

from __future__ import annotations

import argparse
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

CSRC = Path(__file__).resolve().parent
PKG = CSRC.parent
LIB = PKG / "libb200ta.so"
HOST = PKG / "_host.so"
OBJ_DIR = CSRC / "build"
HOST_MADE_FOR = "host_made_for.txt"
SOURCES = ["host.cu", "pack.cu", "rowgemm.cu", "attention.cu", "node.cu", "transition.cu", "trimul_project.cu",
           "trimul_contract.cu", "trimul_output.cu", "linear.cu", "pair_bias.cu", "masks.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo", "--use_fast_math",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libb200ta.so")
    return nvcc


def _deps() -> list[Path]:
    return sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + [PKG.parent / "include" / "b200ta.h"]


def _stale(target: Path, sources: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(s.stat().st_mtime > t for s in sources)


def _host_made_for() -> str:
    """What _host.so depends on besides its sources: the installed PyTorch, whose headers and C++ ABI it is built with, the
    interpreter and the CUDA headers."""
    torch = importlib.util.find_spec("torch")
    return "\n".join([f"torch {importlib.metadata.version('torch')} {Path(torch.origin).parent}", f"python {sys.version}",
                      f"cuda {Path(_nvcc()).resolve().parent.parent}"])


def _host_stale() -> bool:
    """Whether _host.so is missing, older than its sources or made for another PyTorch, interpreter or toolkit."""
    made_for = OBJ_DIR / HOST_MADE_FOR
    return (_stale(HOST, [CSRC / "torch_host.cpp", PKG.parent / "include" / "b200ta.h"])
            or not made_for.exists() or made_for.read_text() != _host_made_for())


def _build_host(force: bool) -> None:
    """_host.so from torch_host.cpp against the headers of the installed PyTorch; it links none of the kernels."""
    if not (force or _host_stale()):
        return
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    cuda = Path(_nvcc()).resolve().parent.parent
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w",
           "-DTORCH_API_INCLUDE_EXTENSION_H", "-DTORCH_EXTENSION_NAME=_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *(f"-I{p}" for p in include_paths()), f"-I{sysconfig.get_paths()['include']}", f"-I{cuda / 'include'}",
           str(CSRC / "torch_host.cpp"), "-o", str(HOST), *(f"-L{p}" for p in library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch_python", f"-L{cuda / 'lib64'}", "-lcudart", "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("building _host.so failed")
    (OBJ_DIR / HOST_MADE_FOR).write_text(_host_made_for())


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ_DIR.mkdir(exist_ok=True)
    sources = [CSRC / s for s in SOURCES if (CSRC / s).exists()]
    deps = _deps()

    def compile_one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        if force or _stale(obj, [src] + deps):
            cmd = [nvcc, *NVCC_FLAGS, *( ["-Xptxas", "-v"] if verbose else []), "-c", str(src), "-o", str(obj)]
            res = subprocess.run(cmd, capture_output=True, text=True)
            if verbose or res.returncode != 0:
                sys.stderr.write(res.stdout + res.stderr)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src.name}")
        return obj

    with ThreadPoolExecutor(max_workers=min(9, len(sources) + 1)) as pool:
        host = pool.submit(_build_host, force)
        objs = list(pool.map(compile_one, sources))
    if force or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-cudart", "static"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("linking libb200ta.so failed")
    host.result()
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
