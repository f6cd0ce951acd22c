"""Builds libq4k_b200.so (CUDA kernels + C ABI) in-tree with nvcc for sm_100a, and the extension through which Python callers reach
its decode entries.  The library needs no Python; without Python's headers (or g++) it is built alone and those entries go through
ctypes."""
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
SOURCES = ["abi.cu", "q8_quantize.cu", "gemv_dp4a.cu", "gemv_mma.cu", "gemv_tma.cu", "mmv_i8.cu", "mmq_mma.cu", "mmq_tcgen05.cu", "mmq_f16.cu", "stream_scratch.cu", "repack.cu", "no_alloc.cu", "peer.cu", "decode_entry.cu", "gemv_bf16w.cu", "fit_q4k.cu", "int8_peak.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return exe


HEADER = PKG.parent / "include" / "q4k_b200.h"


def _stale(target: Path, sources) -> bool:
    return not target.exists() or any(d.stat().st_mtime > target.stat().st_mtime for d in sources)


def library_needs_build() -> bool:
    return _stale(LIB, [d for suffix in ("cu", "cuh", "h") for d in CSRC.glob("*." + suffix)] + [HEADER])


def entries_current() -> bool:
    """The extension is there and no older than what it is built from."""
    return not _stale(ENTRIES, [CSRC / "py_entries.cpp", HEADER])


def entries_buildable() -> bool:
    return shutil.which("g++") is not None and (Path(sysconfig.get_paths()["include"]) / "Python.h").exists()


def needs_build() -> bool:
    return library_needs_build() or (entries_buildable() and not entries_current())


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
            extension = _start_entries() if entries_buildable() and (force or not entries_current()) else None
            if force or library_needs_build():
                _build_library(verbose)
            if extension:
                _finish_entries(*extension)
            return LIB
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def _start_entries():
    tmp = ENTRIES.with_suffix(f".so.tmp{os.getpid()}")
    cmd = ["g++", "-O2", "-std=c++17", "-Wall", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], str(CSRC / "py_entries.cpp"), "-o",
           str(tmp)]
    return tmp, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish_entries(tmp: Path, compiler) -> None:
    out, _ = compiler.communicate()
    if compiler.returncode != 0:
        raise RuntimeError(f"g++ failed on py_entries.cpp:\n{out}")
    os.replace(tmp, ENTRIES)


def _build_library(verbose: bool) -> None:
    objdir = PKG / "lib" / "obj"
    objdir.mkdir(parents=True, exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = objdir / (src + ".o")
        cmd = [nvcc(), *NVCC_FLAGS, "-Xptxas", "-v" if verbose else "-warn-spills", "-c", str(CSRC / src), "-o", str(obj)]
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
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
    os.replace(tmp, LIB)


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
