"""One token of a large MLP chain: gate and up run on dp4a in one launch whose blocks quantise the SwiGLU product."""
import pytest
import torch

from qw38_b200 import q4k_q8_project, synth
from qw38_b200.q4k_q8 import hidden_rms_q8, q4k_q8_mlp, q8_mlp_workspace_bytes, swiglu_pack_q8

pytestmark = pytest.mark.gpu
DEV = "cuda"


# From 2048 super-blocks of eight rows on; an odd number of super-blocks per row group, one; blocks with one group of 32 rows more than others
@pytest.mark.parametrize("hidden,ffn", [(1024, 4096), (768, 11008), (256, 32768), (2048, 4096), (5120, 17408)])
def test_gate_up_pair_quantises_as_the_separate_launches(hidden, ffn):
    gate, up, down = synth.device_weight(ffn, hidden, seed=1), synth.device_weight(ffn, hidden, seed=2), synth.device_weight(hidden, ffn, seed=3)
    g = torch.Generator(device=DEV).manual_seed(hidden)
    h = torch.randn((1, hidden), device=DEV, generator=g) * 2
    gamma = (torch.randn(hidden, device=DEV, generator=g) * 0.1).to(torch.bfloat16)
    flag, other = (torch.zeros(1, dtype=torch.int32, device=DEV) for _ in range(2))
    room = torch.full((q8_mlp_workspace_bytes(1, hidden, ffn),), 77, dtype=torch.uint8, device=DEV)
    out = torch.empty_like(h)

    def run():
        q4k_q8_mlp(gate, up, down, h, gamma, 1e-6, out, 1, room, pending_failure=flag)
        codes, scales = room[:ffn].view(torch.int8), room[ffn:ffn + ffn // 8].view(torch.float32)
        return codes.clone(), scales.clone(), room[ffn + ffn // 8:ffn + ffn // 4].view(torch.int32).clone(), out.clone()

    codes, scales, sums, first = run()
    assert all(torch.equal(a, b) for a, b in zip(run(), (codes, scales, sums, first)))
    x = hidden_rms_q8(h, gamma, 1e-6, other)
    q = swiglu_pack_q8(q4k_q8_project(gate, x), q4k_q8_project(up, x), other)
    # fp32 sums in another order: a product on a bf16 tie moves by one part in 256, and its group's scale with it
    assert (codes.int() - q.codes.view(-1).int()).abs().max() <= 1 and (codes != q.codes.view(-1)).float().mean() < 0.02
    assert ((scales / q.scales.view(-1) - 1).abs() <= 2.0 ** -7).all() and flag.item() == other.item() == 0
    assert torch.equal(sums, codes.view(-1, 32).sum(1).int())
    want = q4k_q8_project(down, q, residual=h)
    assert (first - want).norm() <= 2e-3 * (want - h).norm()
    h[0, hidden // 3] = float("nan")
    _, scales, sums, _ = run()
    assert flag.item() == 1 and torch.isnan(scales).all() and (sums == 0).all()
