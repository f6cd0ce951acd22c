"""Block repack and bf16 decoding at the edges of their tasks: every number of K tiles per warp, ragged rows, and destinations that
are aligned to 16 bytes but not to 32."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from qw38_b200 import _lib as L
from qw38_b200 import synth
from qw38_b200.q4k_q8 import PrefillWeight, pad_n

pytestmark = pytest.mark.gpu


def guarded(count, dtype, offset):
    """`count` elements, `offset` bytes beyond a 256-byte boundary, with the bytes around them."""
    size = count * torch.empty((), dtype=dtype).element_size()
    whole = torch.full((size + 512,), 0x5a, dtype=torch.uint8, device="cuda")
    at = -whole.data_ptr() % 256 + offset
    return whole[at:at + size].view(dtype), whole, at, size


def untouched(whole, at, size):
    return bool((whole[:at] == 0x5a).all()) and bool((whole[at + size:] == 0x5a).all())


@pytest.mark.parametrize("tiles_k", [1, 2, 3, 5, 6, 7, 9, 10, 11, 13, 20, 68])
@pytest.mark.parametrize("n,offset", [(1, 0), (13, 16), (24, 32)])
def test_repack_and_decode(tiles_k, n, offset):
    k = tiles_k * 256
    codes, meta = synth.logical_q4k(n, k, seed=tiles_k + n)
    hc, hs = synth.split_tiles(codes, meta)
    blocks = torch.from_numpy(np.ascontiguousarray(synth.blocks144(codes, meta)).reshape(-1)).cuda()
    pn, lib = pad_n(n), L.load()
    c, cw, ca, cs = guarded(pn * k // 2, torch.uint8, offset)
    s, sw, sa, ss = guarded(pn * tiles_k * 16, torch.uint8, offset)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.q4k_repack_blocks144(vp(blocks), blocks.numel(), n, k, vp(c), c.numel(), vp(s), s.numel(), None) == L.OK
    out, ow, oa, osz = guarded(n * k, torch.bfloat16, offset)
    w = PrefillWeight(c, s, n, k)
    assert lib.q4k_dequantize_bf16(ctypes.byref(w.c_struct()), vp(out), out.numel(), None) == L.OK
    torch.cuda.synchronize()
    assert np.array_equal(c.cpu().numpy(), hc) and np.array_equal(s.cpu().numpy(), hs)
    got = out.view(torch.int16).cpu().numpy().view(np.uint16).reshape(n, k)
    assert np.array_equal(got, orc.dequantize_bf16(codes[:, :k], meta))
    assert untouched(cw, ca, cs) and untouched(sw, sa, ss) and untouched(ow, oa, osz)
