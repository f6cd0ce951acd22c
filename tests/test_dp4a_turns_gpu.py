"""One and two tokens with settled inputs: launches ask for a little more and a little less than half of an SM's shared memory in turn.
Where a run of super-blocks ends inside a ring stage, and where the smaller half holds fewer stages, every launch gives the bits of
the serial one."""
import ctypes

import numpy as np
import pytest
import torch

from qw38_b200 import _lib as L
from qw38_b200 import launch_overlap, pack_q8, q4k_q8_project, set_launch_overlap, synth

pytestmark = pytest.mark.gpu


# stages in either half: the same, two and three, and too few for halves at all
@pytest.mark.parametrize("m,n,k", [(1, 16, 256), (1, 1192, 5120), (2, 2048, 10240), (1, 264, 17408), (2, 1184, 17408), (2, 40, 32768)])
def test_launches_in_turn_give_the_serial_bits(m, n, k):
    w = synth.device_weight(n, k, seed=n)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    x = pack_q8(torch.from_numpy(synth.activations(m, k, seed=k)).cuda(), flag)
    want = q4k_q8_project(w, x, kernel=L.KERNEL_GEMV_DP4A)
    outs = [torch.full_like(want, np.nan) for _ in range(5)]
    torch.cuda.synchronize()
    before = launch_overlap()
    set_launch_overlap(True)
    try:
        for o in outs:
            q4k_q8_project(w, x, out=o, kernel=L.KERNEL_GEMV_DP4A, input_settled=True)
    finally:
        set_launch_overlap(before)
    assert all(torch.equal(o, want) for o in outs) and flag.item() == 0
    status = ctypes.c_int()
    assert L.load().q4k_kernel_status(ctypes.byref(status)) == 0 and status.value == 0
