"""Build libfp8lin.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m "nano-vllm-moe_b200.build"        # or: python nano-vllm-moe_b200/build.py

The shared object is written next to this file so that it travels with the
source tree; nothing is installed into site-packages and nothing is JIT-built
at import time.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OBJ = HERE / "build"
LIB = HERE / "libfp8lin.so"
HOST = HERE / "_fp8host.so"            # the Python binding of the per-step calls (csrc/host.cpp)
SOURCES = ["api.cu", "rmsnorm_quant.cu", "stream_kernel.cu", "elementwise.cu", "umma_gemm.cu", "umma_pair_gemm.cu", "umma_swap.cu", "umma_swap_w8a16.cu", "umma_w8a16_pair.cu", "umma_w8a8_pair.cu", "umma_grouped.cu", "umma_grouped_rows.cu", "umma_grouped_pair.cu", "moe_kernels.cu", "static_scratch.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; the fp8lin library cannot be built")
    return cand


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(d).stat().st_mtime > t for d in deps)


def _compile_host(force: bool) -> tuple[Path, Path]:
    """csrc/host.cpp against this interpreter's and torch's headers; returns the object and torch's library folder."""
    import importlib.util
    root = Path(importlib.util.find_spec("torch").submodule_search_locations[0])
    src, obj = CSRC / "host.cpp", OBJ / "host.cpp.o"
    if force or _stale(obj, [src, HERE.parent / "include" / "fp8lin.h"]):
        cuda = Path(_nvcc()).resolve().parent.parent
        cmd = [shutil.which("g++") or "g++", "-O2", "-fPIC", "-std=c++17", "-fvisibility=hidden", "-D_GLIBCXX_USE_CXX11_ABI=1", "-c", str(src), "-o", str(obj),
               "-isystem", str(root / "include"), "-isystem", str(root / "include" / "torch" / "csrc" / "api" / "include"),
               "-isystem", str(cuda / "include"), "-isystem", sysconfig.get_paths()["include"]]
        r = subprocess.run(cmd, capture_output=True, text=True)
        (OBJ / "host.cpp.log").write_text(r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"g++ failed for host.cpp:\n{r.stdout}\n{r.stderr}")
    return obj, root / "lib"


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ.mkdir(exist_ok=True)
    headers = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + [HERE.parent / "include" / "fp8lin.h"]
    sources = [s for s in SOURCES if (CSRC / s).exists()]

    def compile_one(src: str):
        obj = OBJ / (src + ".o")
        if force or _stale(obj, [CSRC / src, *headers]):
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(CSRC / src), "-o", str(obj)]
            r = subprocess.run(cmd, capture_output=True, text=True)
            (OBJ / (src + ".log")).write_text(r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
            if verbose:
                print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(len(sources) + 1, os.cpu_count() or 1)) as ex:
        host = ex.submit(_compile_host, force)
        objs = list(ex.map(compile_one, sources))
    if force or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    host_obj, torch_lib = host.result()
    if force or _stale(HOST, [host_obj, LIB]):
        cmd = [shutil.which("g++") or "g++", "-shared", "-o", str(HOST), str(host_obj), f"-L{HERE}", "-l:libfp8lin.so", f"-L{torch_lib}", "-ltorch_python",
               "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
