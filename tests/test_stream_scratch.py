"""Per-call scratch (stream_scratch.cu) on the host, over a stand-in for the CUDA runtime."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path("/usr/local/cuda/include")


def test_overlapping_calls_of_a_capture_share_nothing(tmp_path):
    """Calls that alternate, calls that do not (launch overlap switched inside a capture) and calls that fail, in any order:
    a call that is told that it may start early has no byte in common with the one before it."""
    gxx = shutil.which("g++")
    if gxx is None or not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("no g++ or CUDA headers")
    exe = tmp_path / "stream_scratch_check"
    r = subprocess.run([gxx, "-std=c++17", "-O1", "-g", "-fsanitize=address", "-Wall", f"-I{CUDA}", str(ROOT / "tests" / "shim" / "stream_scratch_check.cpp"),
                        "-x", "c++", str(ROOT / "qw38_b200" / "csrc" / "stream_scratch.cu"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, env={"ASAN_OPTIONS": "detect_leaks=0"})
    assert r.returncode == 0 and "stream scratch ok" in r.stdout, r.stdout + r.stderr
