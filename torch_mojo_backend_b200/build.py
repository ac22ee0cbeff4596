"""Ahead-of-time build of ``libb200fa.so`` with nvcc for sm_100a.

Run as ``python -m torch_mojo_backend_b200.build``.  The reference compiles its kernels
lazily on first use and caches the result on disk
(torch_mojo_backend/eager_flash_attention/__init__.py:19-46); here the library is compiled
once, in-tree, before anything runs.  Sources are hashed so an up-to-date library is not
rebuilt.
"""

from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libb200fa.so")
STAMP = os.path.join(HERE, "libb200fa.hash")
SOURCES = ("api.cu", "fwd_sm100.cu", "bwd_sm100.cu", "simt.cu", "simt_bf16.cu", "simt_f16.cu", "decode.cu", "fp32_sm100.cu")
NVCC_FLAGS = (
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared", "--threads", "0",
)


def _source_hash() -> str:
    h = hashlib.sha256()
    names = sorted(os.listdir(CSRC)) + ["../../include/b200fa.h"]
    for name in names:
        path = os.path.normpath(os.path.join(CSRC, name))
        if os.path.isfile(path):
            h.update(name.encode())
            with open(path, "rb") as f:
                h.update(f.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; libb200fa.so cannot be built")
    return nvcc


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library if its sources changed; returns the path of the ``.so``."""
    digest = _source_hash()
    if not force and os.path.exists(LIB) and os.path.exists(STAMP):
        with open(STAMP) as f:
            if f.read().strip() == digest:
                return LIB
    cmd = [find_nvcc(), *NVCC_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB, *[os.path.join(CSRC, s) for s in SOURCES]]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + proc.stdout + proc.stderr)
    with open(STAMP, "w") as f:
        f.write(digest)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
