"""Builds libb200ta.so (sm_100a only) and the layers' native host path (_host.so) next to the package.

Usage: ``python -m bionemo_inference_runtime_b200.csrc.build [--force] [--verbose]``.
The library is linked against the static CUDA runtime and resolves the one
driver symbol it needs at run time, so it loads on machines without a GPU.
"""

from __future__ import annotations

import argparse
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


def _build_host(force: bool) -> None:
    """_host.so from torch_host.cpp against the headers of the installed PyTorch; it links none of the kernels."""
    src = CSRC / "torch_host.cpp"
    if not (force or _stale(HOST, [src, PKG.parent / "include" / "b200ta.h"])):
        return
    import sysconfig

    from torch.utils.cpp_extension import include_paths, library_paths

    cuda = Path(_nvcc()).resolve().parent.parent
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w",
           "-DTORCH_API_INCLUDE_EXTENSION_H", "-DTORCH_EXTENSION_NAME=_host", "-D_GLIBCXX_USE_CXX11_ABI=1",
           *(f"-I{p}" for p in include_paths()), f"-I{sysconfig.get_paths()['include']}", f"-I{cuda / 'include'}",
           str(src), "-o", str(HOST), *(f"-L{p}" for p in library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch_python", f"-L{cuda / 'lib64'}", "-lcudart", "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("building _host.so failed")


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
