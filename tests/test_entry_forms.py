"""The decode entries reach C through the extension or, where that was not built, through ctypes: the same calls with the same
arguments, and a library named by Q4K_B200_LIBRARY or a box without Python's headers needs nothing else."""
import ctypes as C
import os
import subprocess
import sys
import types
from pathlib import Path

import pytest
import torch

from qw38_b200 import _lib as L
from qw38_b200 import build
from qw38_b200._entries import CtypesEntries
from qw38_b200.q4k_q8 import DecodeMmvDesc, PrefillWeight, Q8Input

ROOT = Path(__file__).resolve().parents[1]
NAMES = ("decode_mmv", "decode_mmv_ranges", "pack_q8_bf16", "pack_q8_f32", "q8_project", "q8_mlp", "prefill_project", "prefill_paired_swiglu",
         "decode_mmv_paired")


class Stream:
    cuda_stream = 4321


def plain(value):
    """An argument as bytes or a number: structures by content, without the padding at the end of a descriptor."""
    if isinstance(value, C._Pointer):
        value = value.contents
    if isinstance(value, C.Structure):
        return bytes(value)[:-2] if isinstance(value, L.DecodeDesc) else bytes(value)
    return value


@pytest.fixture
def forms():
    """Both forms bound to functions that record what reaches the C entry; q8_mlp also reports `submitted`."""
    calls = []

    def recorder(name):
        res, args = L.SIGNATURES["q4k_" + name]

        def f(*got):
            if name == "decode_mmv_ranges":
                calls.append((name, [plain(got[0][i]) for i in range(min(got[1], 3))], *got[1:]))
            elif name == "q8_mlp":
                calls.append((name, *(plain(v) for v in got[:11]), got[12]))
                got[11][0] = 1
            else:
                calls.append((name, *(plain(v) for v in got)))
            return 3

        return C.CFUNCTYPE(res, *args)(f)

    fakes = {n: recorder(n) for n in NAMES}
    lib, module = L.load(), L.entries()
    if isinstance(module, CtypesEntries):
        pytest.skip("no extension on this box")
    real = [C.cast(getattr(lib, "q4k_" + n), C.c_void_p).value for n in NAMES]
    module.bind(*(C.cast(fakes[n], C.c_void_p).value for n in NAMES), torch._C._cuda_getDevice, torch._C._cuda_getCurrentRawStream)
    yield module, CtypesEntries(types.SimpleNamespace(**{"q4k_" + n: f for n, f in fakes.items()}), L.DecodeDesc), calls
    module.bind(*real, torch._C._cuda_getDevice, torch._C._cuda_getCurrentRawStream)


def weight(n, k):
    pn, pk = (n + 7) // 8 * 8, (k + 255) // 256 * 256
    return PrefillWeight(torch.zeros(pn * pk // 2, dtype=torch.uint8), torch.zeros(pn * pk // 16, dtype=torch.uint8), n, k)


def test_both_forms_make_the_same_calls(forms):
    module, other, calls = forms
    w, v = weight(40, 300), weight(13, 300)
    x, out, res = torch.zeros((3, 300), dtype=torch.bfloat16), torch.zeros((3, 40)), torch.zeros((3, 40))
    q = Q8Input(torch.zeros((3, 512), dtype=torch.int8), torch.zeros((3, 16)), torch.zeros((3, 16), dtype=torch.int32), 3, 300, 512)
    d, e = DecodeMmvDesc(w, x, out, L.EPILOGUE_RESIDUAL_ADD_FP32, res), DecodeMmvDesc(v, x[0], None)
    ws, wide, f, s = torch.zeros(512, dtype=torch.uint8), torch.zeros(64), torch.zeros(1, dtype=torch.int32), Stream()
    gamma = torch.zeros(300, dtype=torch.bfloat16)
    for name, args in [("decode_mmv", (d, ws, f, s)), ("decode_mmv", (e, ws, None, s)), ("prefill_project", (d, ws, f, s)),
                       ("decode_mmv_ranges", ([d, e], ws, f, s)), ("decode_mmv_ranges", ((d, e, d), ws, f, s)),
                       ("decode_mmv_ranges", ([], ws, f, s)), ("decode_mmv_ranges", ([d] * 5, ws, f, s)),
                       ("decode_mmv_paired", (d, e, ws, f, s)), ("decode_mmv_paired", (e, d, ws, None, s)),
                       ("prefill_paired_swiglu", (w, v, x, out, 3, ws, f, s)), ("pack_q8", (x, False, q, f, s)), ("pack_q8", (res, True, q, f, s)),
                       ("q8_project", (w, q, out, None, s)), ("q8_project", (w, q, out, res, s)),
                       ("q8_mlp", (w, v, w, res, gamma, 1e-6, out, 3, wide, f, s)), ("q8_mlp", (w, v, w, res, gamma, 1e-6, out, 3, wide, None, s))]:
        del calls[:]
        results = [getattr(form, name)(*args) for form in (module, other)]
        assert results[0] == results[1] == ((3, 1) if name == "q8_mlp" else 3)
        assert len(calls) == 2 and calls[0] == calls[1], name


PROBE = """
import torch
from qw38_b200 import _lib as L, build
from qw38_b200._entries import CtypesEntries
{setup}
from qw38_b200.q4k_q8 import DecodeMmvDesc, PrefillWeight, Q4KError, launch_decode_mmv
L.load()
print(type(L.entries()).__name__, build.needs_build())
class Stream:
    cuda_stream = 0
w = PrefillWeight(torch.zeros(1024, dtype=torch.uint8), torch.zeros(128, dtype=torch.uint8), 8, 256, layout=1)
try:
    launch_decode_mmv(DecodeMmvDesc(w, torch.zeros((1, 256), dtype=torch.bfloat16), torch.zeros((1, 8))), torch.zeros(64, dtype=torch.uint8),
                      torch.zeros(1, dtype=torch.int32), Stream)
except Q4KError as e:
    print(e.code)
"""


def run(setup="", **env):
    r = subprocess.run([sys.executable, "-c", PROBE.format(setup=setup)], cwd=ROOT, env={**os.environ, **env}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return r.stdout.split()


NEVER_BUILT = "build.ENTRIES = build.LIB.with_name('_q4k_entries_missing.so')"


def test_a_named_library_needs_no_extension(tmp_path):
    named = tmp_path / "libq4k_b200.so"
    named.symlink_to(build.build())
    assert run(NEVER_BUILT, Q4K_B200_LIBRARY=str(named))[::2] == ["CtypesEntries", str(L.ERR_INVALID_ARGUMENT)]


@pytest.mark.parametrize("content", ["the package's", "no extension"])
def test_the_extension_beside_a_named_library_is_used(tmp_path, content):
    named = tmp_path / "libq4k_b200.so"
    named.symlink_to(build.build())
    if content == "no extension":
        (tmp_path / build.ENTRIES.name).write_bytes(b"of another interpreter")
    elif build.entries_current():
        (tmp_path / build.ENTRIES.name).symlink_to(build.ENTRIES)
    kind = "module" if content != "no extension" and build.entries_current() else "CtypesEntries"
    assert run(Q4K_B200_LIBRARY=str(named))[::2] == [kind, str(L.ERR_INVALID_ARGUMENT)]


@pytest.mark.parametrize("missing", ["sysconfig.get_paths = lambda: {'include': '/nonexistent'}",
                                     "shutil.which = lambda name, which=shutil.which: None if name == 'g++' else which(name)"])
def test_a_box_that_cannot_build_the_extension_builds_the_library(missing):
    build.build()
    assert run(f"import shutil, sysconfig\n{NEVER_BUILT}\n{missing}") == ["CtypesEntries", "False", str(L.ERR_INVALID_ARGUMENT)]
