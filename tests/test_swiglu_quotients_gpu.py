"""silu() of the SwiGLU pack and sigmoid_fp32() of the SwiGLU store are computed through one reciprocal and a residual correction:
the bits of the divisions for all 2^32 arguments, but for the sign of the pack's quotient of -0."""
import subprocess
from pathlib import Path

import pytest

from qw38_b200 import build

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.gpu
def test_quotients_are_the_divisions(tmp_path):
    exe = tmp_path / "swiglu_quotients"
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, str(ROOT / "tests" / "shim" / "swiglu_quotients.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
