"""Builds libq4k_b200.so (CUDA kernels + C ABI) in-tree with nvcc for sm_100a."""
from __future__ import annotations

import os
import shutil
import subprocess
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "lib" / "libq4k_b200.so"
ENTRIES = PKG / "lib" / "_q4k_entries.so"  # Python's way into the entries of a decode step (csrc/py_entries.cpp)
SOURCES = ["abi.cu", "q8_quantize.cu", "gemv_dp4a.cu", "gemv_mma.cu", "gemv_tma.cu", "mmq_mma.cu", "mmq_tcgen05.cu", "mmq_f16.cu", "stream_scratch.cu", "repack.cu", "no_alloc.cu", "peer.cu", "decode_entry.cu", "gemv_bf16w.cu", "fit_q4k.cu", "int8_peak.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return exe


def needs_build() -> bool:
    if not LIB.exists() or not ENTRIES.exists():
        return True
    t = min(LIB.stat().st_mtime, ENTRIES.stat().st_mtime)
    deps = list(CSRC.glob("*.cpp")) + list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + \
        [PKG.parent / "include" / "q4k_b200.h"]
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every kernel file to objects in parallel and link the shared library.

    Several processes may import the package at once (one rank per GPU): the check and the build run under
    an exclusive file lock, and the library is linked under a temporary name and renamed into place, so a
    rank either waits for the one that builds or finds a complete library."""
    import fcntl
    LIB.parent.mkdir(parents=True, exist_ok=True)
    with open(LIB.parent / ".build.lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not needs_build():
                return LIB
            return _build_locked(verbose)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def _build_locked(verbose: bool) -> Path:
    objdir = PKG / "lib" / "obj"
    objdir.mkdir(parents=True, exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = objdir / (src + ".o")
        cmd = [nvcc(), *NVCC_FLAGS, "-Xptxas", "-v" if verbose else "-warn-spills", "-c", str(CSRC / src), "-o", str(obj)]
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    entries = ENTRIES.with_suffix(f".so.tmp{os.getpid()}")
    cmd = ["g++", "-O2", "-std=c++17", "-Wall", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], str(CSRC / "py_entries.cpp"), "-o",
           str(entries)]
    host = subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    objs = []
    for src, obj, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose:
            print(out)
        objs.append(str(obj))
    tmp = LIB.with_suffix(f".so.tmp{os.getpid()}")
    cmd = [nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(tmp), *objs]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}{r.stderr}")
    out, _ = host.communicate()
    if host.returncode != 0:
        raise RuntimeError(f"g++ failed on py_entries.cpp:\n{out}")
    os.replace(entries, ENTRIES)
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
