"""Build recipe of the CUDA library (in-tree, sm_100a only).

    python -m camellia2_b200.build      # -> camellia2_b200/libdpg_b200.so
"""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = [os.path.join(HERE, "csrc", f"dpg_{f}.cu") for f in ("host", "kernel", "small", "queue", "adjoint", "energy", "big", "maps")]
OUT = os.path.join(HERE, "libdpg_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def build(verbose=False):
    flags = FLAGS + (["-Xptxas", "-v"] if verbose else [])
    with tempfile.TemporaryDirectory() as tmp:  # one nvcc per translation unit, side by side
        objs = [os.path.join(tmp, os.path.basename(f) + ".o") for f in SRC]
        jobs = [subprocess.Popen([NVCC] + flags + ["-c", f, "-o", o]) for f, o in zip(SRC, objs)]
        if any([j.wait() for j in jobs]):
            raise RuntimeError("nvcc failed")
        subprocess.check_call([NVCC] + flags + ["-shared"] + objs + ["-o", OUT, "-lcudart"])
    return OUT


if __name__ == "__main__":
    build(verbose="-v" in sys.argv)
    print(OUT)
