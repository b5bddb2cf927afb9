"""Build the in-tree CUDA library ``gegs_b200/libgegs_b200.so`` for sm_100a.

The library is compiled with ``-fmad=false`` (no FMA contraction) and IEEE
division / square root, which together with the library's own transcendental
functions makes every particle history reproducible bit for bit.
"""
from __future__ import annotations

import os
import pathlib
import subprocess
import tempfile

PKG = pathlib.Path(__file__).resolve().parent
SRC = PKG / "csrc"
INC = PKG.parent / "include"
LIB = PKG / "libgegs_b200.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-fmad=false", "-prec-div=true", "-prec-sqrt=true", "-ftz=false",
    "-Xcompiler", "-fPIC",
]


def sources():
    return sorted(list(SRC.glob("*.cu")) + list(SRC.glob("*.cuh")) + list(SRC.glob("*.cpp")) + list(SRC.glob("*.h"))
                  + list(INC.glob("*.h")))


def needs_build() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    return any(s.stat().st_mtime > t for s in sources())


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    if not force and not needs_build():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    units = sorted(list(SRC.glob("*.cu")) + list(SRC.glob("*.cpp")))
    flags = [*(["-Xptxas=-v"] if verbose else []), *NVCC_FLAGS, "-Xcompiler", "-ffp-contract=off"]
    with tempfile.TemporaryDirectory() as tmp:
        # the translation units side by side: each holds kernels that take a minute or two
        objs = [pathlib.Path(tmp) / (u.name + ".o") for u in units]
        jobs = [subprocess.Popen([nvcc, *flags, "-c", str(u), "-o", str(o)]) for u, o in zip(units, objs)]
        for u, j in zip(units, [j.wait() for j in jobs]):
            if j != 0:
                raise subprocess.CalledProcessError(j, f"nvcc -c {u}")
        out = LIB.with_suffix(".so.tmp")
        subprocess.run([nvcc, *NVCC_FLAGS, "-shared", "-o", str(out), *map(str, objs)], check=True)
    os.replace(out, LIB)
    return LIB


if __name__ == "__main__":
    import sys
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
