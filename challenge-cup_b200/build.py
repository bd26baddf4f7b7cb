"""Build the in-tree CUDA library ``ertm_b200/libertm_b200.so`` for sm_100a.

    python challenge-cup_b200/build.py [--verbose-ptxas]

nvcc cross-compiles without a GPU.  The shared library is written next to
the Python package so it travels with the repository snapshot.
"""

from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OUT = HERE / "ertm_b200" / "libertm_b200.so"
SOURCES = [CSRC / "ertm_b200.cu", CSRC / "wave.cu"]
DEPS = sorted(CSRC.glob("*.cu*")) + sorted(CSRC.glob("*.h")) + [HERE.parent / "include" / "ertm_b200.h"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc() -> str:
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    path = Path(cuda) / "bin" / "nvcc"
    return str(path) if path.exists() else "nvcc"


def up_to_date() -> bool:
    if not OUT.exists():
        return False
    built = OUT.stat().st_mtime
    return all(p.stat().st_mtime <= built for p in DEPS + [Path(__file__)])


def build(force: bool = False, ptxas_verbose: bool = False) -> Path:
    if not force and up_to_date():
        return OUT
    flags = [*ARCH, "-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC,-O3"]
    if ptxas_verbose:
        flags.append("-Xptxas=-v")
    # the translation units compile side by side; objects and the new library
    # have names of their own, so builds do not meet and failures leave nothing
    tmp = OUT.with_suffix(f".so.{os.getpid()}.tmp")
    with tempfile.TemporaryDirectory(prefix="ertm-build-") as d:
        objects = [Path(d) / f"{src.stem}.o" for src in SOURCES]
        procs = [subprocess.Popen([nvcc(), *flags, "-c", "-o", str(obj), str(src)], stdout=subprocess.PIPE,
                                  stderr=subprocess.STDOUT, text=True) for src, obj in zip(SOURCES, objects)]
        logs = [p.communicate()[0] for p in procs]
        for p, log in zip(procs, logs):
            if p.returncode != 0 or ptxas_verbose:
                sys.stderr.write(log)
        if any(p.returncode != 0 for p in procs):
            raise RuntimeError("nvcc failed")
        link = [nvcc(), *ARCH, "-shared", "-o", str(tmp), *map(str, objects), "-lcufft"]
        res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        tmp.unlink(missing_ok=True)
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError(f"nvcc (link) failed with exit code {res.returncode}")
    os.replace(tmp, OUT)
    return OUT


if __name__ == "__main__":
    p = build(force=True, ptxas_verbose="--verbose-ptxas" in sys.argv)
    print(p)
