"""Build ``libb2kv.so`` (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

``python llm-experiments_b200/build.py [--force] [--verbose] [--serve]``.  The library has no
dependency on torch or Python: it is loaded with ctypes.  Sources are compiled to
objects in parallel and linked with the static CUDA runtime.

``--serve`` builds ``libb2kv_serve.so`` instead: only what models with a 32-bit residual stream are served with, a
fraction of the compile time (the decode-attention and prefill variants of the reference path take most of it).  It is
loaded where the whole library has not been built.
"""
from __future__ import annotations

import concurrent.futures
import os
import pathlib
import platform
import subprocess
import sys
import sysconfig

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
OUT = PKG / "libb2kv.so"
CALLS = PKG / ("b2kv_calls" + sysconfig.get_config_var("EXT_SUFFIX"))  # the C ABI's calls from Python, for this interpreter alone
SERVE_OUT = PKG / "libb2kv_serve.so"
OBJ_DIR = PKG / "build"
SERVE_SOURCES = ("api", "append", "gemm", "gla", "gla_chunked", "gla_run", "gqa", "gqa_decode_tc", "latent", "latent_decode_tc", "latent_prefill", "linear", "linear_f32", "linear_f32_tc", "linear_rows", "moe", "rows",
                 "step_tail")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else "nvcc"


def sources(serve: bool = False):
    return [f for f in sorted(CSRC.glob("*.cu")) if not serve or f.stem in SERVE_SOURCES]


def _newest_input() -> float:
    files = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    return max(f.stat().st_mtime for f in files)


def up_to_date(out: pathlib.Path = OUT) -> bool:
    return out.exists() and out.stat().st_mtime >= _newest_input()


def build_calls(force: bool = False) -> None:
    """The extension module of ``csrc/calls.c`` with the C compiler.  The library does without it (ctypes makes the calls then), so
    where it cannot be built there is a note and no error."""
    src, include = CSRC / "calls.c", pathlib.Path(sysconfig.get_paths()["include"])
    if not force and CALLS.exists() and CALLS.stat().st_mtime >= src.stat().st_mtime:
        return
    why = None
    if sys.platform != "linux" or platform.machine() != "x86_64":
        why = "its calls are those of x86-64 Linux"
    elif not (include / "Python.h").exists():
        why = "there are no headers of this interpreter"
    else:
        cmd = [os.environ.get("CC", "gcc"), "-O2", "-Wall", "-shared", "-fPIC", "-I", str(include), str(src), "-o", str(CALLS)]
        try:
            res = subprocess.run(cmd, capture_output=True, text=True)
            if res.returncode != 0:
                why = f"{cmd[0]} failed: {res.stderr.strip()}"
        except OSError as e:
            why = str(e)
    if why is not None:
        CALLS.unlink(missing_ok=True)  # (one of an older source)
        sys.stderr.write(f"{CALLS.name} is not built, calls go through ctypes: {why}\n")


def build(force: bool = False, verbose: bool = False, serve: bool = False) -> pathlib.Path:
    build_calls(force)
    out = SERVE_OUT if serve else OUT
    if not force and up_to_date(out):
        return out
    OBJ_DIR.mkdir(exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: pathlib.Path) -> pathlib.Path:
        obj = OBJ_DIR / (src.stem + ".o")
        cmd = [_nvcc(), *NVCC_FLAGS, *extra, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}")
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, sources(serve)))
    link = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(out), *map(str, objs)]
    subprocess.run(link, check=True)
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, serve="--serve" in sys.argv))
