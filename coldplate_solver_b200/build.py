"""Build recipe for libcps.so (sm_100a) -- compiled in-tree so it travels with
the repository snapshot.

The tile shape of the kernels is a compile-time constant, so each shape is
its own library with the same C ABI: libcps.so (8 x 32 tiles, the default and
the one the C++ drop-in links), libcps_t16.so (16 x 16) and libcps_t64.so
(4 x 64).  Their sources compile in parallel.

``--fmad=false``: the FP64 path keeps the reference's separate multiply and
add roundings, so per-point values match the FP64 reference exactly; the
kernels are bound by memory and barrier latency, not by FP64 issue rate.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
import tempfile

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
REPO_DIR = os.path.dirname(PKG_DIR)
LIB_PATH = os.path.join(PKG_DIR, "libcps.so")
TILE_WIDTHS = (32, 16, 64)  # tile columns; rows = 256 / columns


def lib_path(tile_j: int = 32) -> str:
    """The library built with tiles of ``tile_j`` columns."""
    if tile_j not in TILE_WIDTHS:
        raise ValueError(f"tile width {tile_j} is not built (have {TILE_WIDTHS})")
    return LIB_PATH if tile_j == 32 else os.path.join(PKG_DIR, f"libcps_t{tile_j}.so")


SOURCES = [os.path.join(PKG_DIR, "csrc", f) for f in (
    "cps_grid_f64.cu", "cps_grid_f32.cu", "cps_grid_opt_f64.cu", "cps_grid_opt_f32.cu", "cps_grid_mon_f64.cu",
    "cps_grid_mon_f32.cu", "cps_batch_f64.cu", "cps_batch_f32.cu", "cps_batch_opt_f64.cu", "cps_batch_opt_f32.cu",
    "cps_api.cu", "cps_noalloc.cu", "cps_thermal.cu", "cps_io.cpp", "cps_thermal_io.cpp")]
HEADERS = [os.path.join(PKG_DIR, "csrc", f) for f in os.listdir(os.path.join(PKG_DIR, "csrc")) if f.endswith((".cuh", ".h"))]
HEADERS.append(os.path.join(REPO_DIR, "include", "cps.h"))
HEADERS.append(os.path.join(REPO_DIR, "include", "cps_thermal.h"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "--fmad=false", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared",
    "-static-global-template-stub=false",  # kernels are instantiated in files of their own
]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def needs_build(path: str = LIB_PATH) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(f) > t for f in SOURCES + HEADERS)


def build(force: bool = False, verbose: bool = False) -> str:
    """Build every tile-shape library that is missing or older than its
    sources (all of them with ``force``); returns the default library's path."""
    todo = [j for j in TILE_WIDTHS if force or needs_build(lib_path(j))]
    env = dict(os.environ)
    env.pop("CXX", None)
    env.pop("CC", None)
    flags = [f for f in NVCC_FLAGS if f != "-shared"] + (["-Xptxas=-v"] if verbose else [])
    with tempfile.TemporaryDirectory() as tmp, concurrent.futures.ThreadPoolExecutor(os.cpu_count()) as pool:
        def compile_one(j: int, src: str):
            obj = os.path.join(tmp, f"{os.path.basename(src)}.{j}.o")
            cmd = [nvcc(), *flags, f"-DCPS_TILE_J={j}", "-c", "-o", obj, src]
            if verbose:
                print(" ".join(cmd), file=sys.stderr)
            return obj, subprocess.run(cmd, env=env).returncode

        jobs = {j: [pool.submit(compile_one, j, src) for src in SOURCES] for j in todo}
        for j, futures in jobs.items():
            objs = [f.result() for f in futures]
            if any(rc for _, rc in objs) or subprocess.run(
                    [nvcc(), *NVCC_FLAGS, "-o", lib_path(j), *[o for o, _ in objs]], env=env).returncode:
                raise RuntimeError(f"nvcc failed for tile width {j}")
    return LIB_PATH


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
