"""One token from bf16 rows: two dp4a blocks per SM share the row groups of eight.  Counts around one and two blocks per SM (148 SMs),
a ragged last group, fewer groups than blocks, several matrices in one launch, and rows that take no 16-byte loads."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from qw38_b200 import _lib as L
from qw38_b200 import synth
from qw38_b200.q4k_q8 import DecodeMmvDesc, PrefillWeight, decode_workspace, launch_decode_mmv, launch_decode_mmv_ranges
from tests.helpers import assert_close_contract

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [(3,), (1184,), (1185,), (2368,), (2376,), (4741,), (1184, 8, 1177)])
@pytest.mark.parametrize("k", [256, 1003])
def test_row_groups_over_two_blocks_per_sm(rows, k):
    x = torch.from_numpy(synth.activations(1, k, seed=k)).to(DEV).to(torch.bfloat16)
    z, a, s, _ = orc.q8_quantize(x.view(torch.int16).cpu().numpy().view(np.uint16), bf16_bits=True)
    parts = []
    for i, n in enumerate(rows):
        codes, meta = synth.logical_q4k(n, k, seed=n + i)
        hc, hs = synth.split_tiles(codes, meta)
        parts.append((PrefillWeight.from_host(hc, hs, n, k), hc, hs, torch.empty((1, n), dtype=torch.float32, device=DEV)))
    f = torch.zeros(1, dtype=torch.int32, device=DEV)
    descs, ws = [DecodeMmvDesc(w, x, out, L.EPILOGUE_STORE_FP32) for w, _, _, out in parts], decode_workspace(1, sum(rows), k)
    if len(descs) > 1:
        launch_decode_mmv_ranges(descs, ws, f)
    else:
        launch_decode_mmv(descs[0], ws, f)
    status = ctypes.c_int(-1)
    assert L.load().q4k_kernel_status(ctypes.byref(status)) == 0 and status.value == 0 and f.item() == 0
    for w, hc, hs, out in parts:
        assert_close_contract(out.cpu().numpy(), orc.project(hc, hs, w.n, w.padded_k, z, a, s))
