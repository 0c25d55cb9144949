"""Builds libb200lm.so (sm_100a only) next to this file with nvcc.

    python litert-lm_b200/build.py [--force]

The shared library is self-contained (static CUDA runtime) and exports the C ABI
declared in include/b200lm.h and include/b200lm_ops.h.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200lm.so")
# one translation unit per kernel family and cache type, compiled side by side
SOURCES = ["lib.cu", "decode_step.cu"] + [f"{k}_{t}.cu" for k in ("decode_stream", "decode_wide", "attn_mma") for t in ("f32", "bf16")]


def _deps():
    """Every file the translation unit can include."""
    inc = os.path.join(HERE, "..", "include")
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    files += [os.path.join(inc, f) for f in os.listdir(inc) if f.endswith(".h")]
    return files


def nvcc_path() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(d) > t for d in _deps())


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC,-O2"]
    if verbose:
        flags.insert(0, "-Xptxas=-v")
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    nvcc = nvcc_path()

    def run(cmd) -> None:
        res = subprocess.run(cmd, capture_output=True, text=True, env=env)
        if res.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
        if verbose:
            print(res.stderr)

    with tempfile.TemporaryDirectory() as tmp:
        objs = [os.path.join(tmp, s + ".o") for s in SOURCES]
        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
            list(pool.map(run, [[nvcc] + flags + ["-c", os.path.join(CSRC, s), "-o", o] for s, o in zip(SOURCES, objs)]))
        run([nvcc] + flags + ["-shared", "-o", LIB] + objs)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
