"""The extension through which Python callers reach the decode entries reads what the ctypes structures say: the same structure
for plain, overridden and malformed descriptors, and errors instead of crashes for objects of another kind."""
import ctypes as C

import numpy as np
import pytest
import torch

from qw38_b200 import _lib as L
from qw38_b200.q4k_q8 import DecodeMmvDesc, PrefillWeight, new_q8_input

NAMES = ("decode_mmv", "decode_mmv_ranges", "pack_q8_bf16", "pack_q8_f32", "q8_project", "q8_mlp", "prefill_project", "prefill_paired_swiglu")


class Stream:
    cuda_stream = 1234


@pytest.fixture
def probe():
    """The extension bound to a function that records the bytes behind its first argument."""
    seen = {}
    kinds = {"desc": C.sizeof(L.DecodeDesc), "weight": C.sizeof(L.Weight)}

    def recorder(name, size):
        def f(first, a, b, c, d):
            seen[name] = (C.string_at(first, size), a, b, c, d)
            return 7
        return C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_uint64, C.c_void_p, C.c_void_p)(f)

    lib, module = L.load(), L.entries()
    real = [C.cast(getattr(lib, "q4k_" + n), C.c_void_p).value for n in NAMES]
    one = recorder("one", kinds["desc"])
    fakes = list(real)
    fakes[0] = fakes[6] = C.cast(one, C.c_void_p).value
    module.bind(*fakes, lambda: 0, lambda device: 99)
    yield module, seen
    module.bind(*real, torch._C._cuda_getDevice, torch._C._cuda_getCurrentRawStream)


def weight(n, k, **more):
    pn, pk = (n + 7) // 8 * 8, (k + 255) // 256 * 256
    return PrefillWeight(torch.zeros(pn * pk // 2, dtype=torch.uint8), torch.zeros(pn * pk // 16, dtype=torch.uint8), n, k, **more)


@pytest.mark.parametrize("case", ["plain", "one row", "no output", "overridden", "malformed"])
def test_descriptors_are_the_ctypes_ones(probe, case):
    module, seen = probe
    w = weight(40, 300)
    x, out, res = torch.zeros((3, 300), dtype=torch.bfloat16), torch.zeros((3, 40)), torch.zeros((3, 40))
    d = DecodeMmvDesc(w, x, out, L.EPILOGUE_RESIDUAL_ADD_FP32, res)
    if case == "one row":
        d = DecodeMmvDesc(w, x[0], out[0])
    elif case == "no output":
        d = DecodeMmvDesc(w, x, None, L.EPILOGUE_RESIDUAL_ADD_FP32, res)
    elif case == "overridden":
        d.weight = weight(40, 300, codes_bytes=5, scales_bytes=6)
    elif case == "malformed":
        d.weight.layout, d.weight.quantizer, d.epilogue, d.activation_policy = 70000, 3, 260, 255
    ws, f = torch.zeros(512, dtype=torch.uint8), torch.zeros(1, dtype=torch.int32)
    for call in (module.decode_mmv, module.prefill_project):
        for stream, handle in ((None, 99), (Stream(), 1234)):
            assert call(d, ws, f, stream) == 7
            got, a, b, c, s = seen["one"]  # (two bytes of padding at the end)
            want = bytes(d.c_struct())
            assert got[:-2] == want[:-2] and (a, b, c, s) == (ws.data_ptr(), 512, f.data_ptr(), handle)
    assert module.decode_mmv(d, ws, None, None) == 7 and seen["one"][3] is None


def test_other_objects_raise(probe):
    module, _ = probe
    w = weight(8, 256)
    d = DecodeMmvDesc(w, torch.zeros((1, 256), dtype=torch.bfloat16), torch.zeros((1, 8)))
    ws, f = torch.zeros(8, dtype=torch.uint8), torch.zeros(1, dtype=torch.int32)
    with pytest.raises(TypeError):
        module.decode_mmv(d, ws, f)
    with pytest.raises(AttributeError):
        module.decode_mmv(object(), ws, f, None)
    with pytest.raises(AttributeError):
        module.decode_mmv(d, None, f, None)
    with pytest.raises(TypeError):
        module.decode_mmv_ranges(5, ws, f, None)
    with pytest.raises(AttributeError):
        module.q8_project(w, new_q8_input(1, 256, device="cpu"), None, None, None)
    with pytest.raises(TypeError):
        module.q8_mlp(w, w, w, f, f, "eps", f, 1, ws, None, None)
    w.n = "eight"
    with pytest.raises(TypeError):
        module.decode_mmv(d, ws, f, None)


class Index:
    """An integer by __index__ alone."""

    def __init__(self, value):
        self.value = value

    def __index__(self):
        return self.value


@pytest.mark.parametrize("kind", [np.int64, np.int32, np.uint16, np.uint64, Index])
def test_integers_of_other_types_are_taken(probe, kind):
    """Shapes come from numpy and file headers: everything with __index__ is an integer here as in the ctypes structures."""
    module, seen = probe
    w = weight(40, 512)
    want = bytes(DecodeMmvDesc(w, torch.zeros((1, 512), dtype=torch.bfloat16), None).c_struct())
    x = torch.zeros((1, 512), dtype=torch.bfloat16)
    d = DecodeMmvDesc(weight(40, 512), x, None)
    d.weight.codes, d.weight.scales = w.codes, w.scales
    d.weight.n, d.weight.k, d.weight.layout, d.weight.quantizer = kind(40), kind(512), kind(w.layout), kind(w.quantizer)
    d.weight.codes_bytes, d.weight.scales_bytes = kind(w.codes.numel()), kind(w.scales.numel())
    d.epilogue, d.activation_policy = kind(d.epilogue), kind(d.activation_policy)
    ws, f = torch.zeros(512, dtype=torch.uint8), torch.zeros(1, dtype=torch.int32)
    assert module.decode_mmv(d, ws, f, None) == 7
    got, at = seen["one"][0], L.DecodeDesc.input.offset
    assert got[:at] == want[:at] and got[at + 8:-2] == want[at + 8:-2]  # (all but the address of the other input)
    # the counts that are arguments of their own, refused by the library before it looks at anything else
    w.layout = 0
    lib, m = L.load(), kind(3)
    q = new_q8_input(3, 512, device="cpu")
    q.m, q.k, q.padded_k = kind(3), kind(512), kind(512)
    for call in (lambda: module.q8_mlp(w, w, w, f, f, 1e-6, f, m, ws, f, None)[0],
                 lambda: module.prefill_paired_swiglu(w, w, x, x, m, ws, f, None), lambda: module.q8_project(w, q, f, None, None)):
        assert call() == L.ERR_INVALID_ARGUMENT and lib.q4k_last_error()
    for bad in (8.0, np.float32(8), "8", None):
        d.weight.n = bad
        with pytest.raises(TypeError):
            module.decode_mmv(d, ws, f, None)


@pytest.mark.parametrize("shrink", [list.clear, lambda ranges: ranges.__delitem__(slice(1, None))])
def test_a_list_that_shrinks_while_it_is_read(probe, shrink):
    """Reading a descriptor runs Python code, which may change the list of ranges: what the list held at the call counts."""
    module, _ = probe
    w = weight(8, 256)
    w.layout = 0  # refused before any device work

    class Shrinking(DecodeMmvDesc):
        @property
        def epilogue(self):
            shrink(ranges)
            return L.EPILOGUE_STORE_FP32

        @epilogue.setter
        def epilogue(self, value):
            pass

    x, ws, f = torch.zeros((1, 256), dtype=torch.bfloat16), torch.zeros(8, dtype=torch.uint8), torch.zeros(1, dtype=torch.int32)
    for _ in range(200):  # (the other descriptors live in the list alone)
        ranges = [Shrinking(w, x, torch.zeros((1, 8))), DecodeMmvDesc(w, x, torch.zeros((1, 8))), DecodeMmvDesc(w, x, torch.zeros((1, 8)))]
        assert module.decode_mmv_ranges(ranges, ws, f, None) == L.ERR_INVALID_ARGUMENT
        assert len(ranges) <= 1
