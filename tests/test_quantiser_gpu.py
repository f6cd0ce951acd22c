"""The quantiser's scale and quotients come from reciprocals: bitwise the divisions, for every mantissa of the peak at both ends of
the range that takes this path, beyond them, and for values that are not finite."""
import pytest
import torch

from qw38_b200.q4k_q8 import pack_q8

pytestmark = pytest.mark.gpu


def check(x, flagged):
    f = torch.zeros(1, dtype=torch.int32, device="cuda")
    q = pack_q8(x, f)
    g = x.view(-1, 32)
    finite = torch.isfinite(g).all(1)
    peak = g.abs().amax(1)
    a = torch.where(peak == 0, torch.ones_like(peak), peak / torch.full_like(peak, 127.0))  # (a scalar divisor would be inverted)
    valid = finite & (a > 0)
    z = torch.where(valid[:, None], torch.clamp(torch.round(g / a[:, None]), -127, 127), torch.zeros_like(g))
    assert torch.equal(q.codes.view(-1, 32), z.to(torch.int8)) and torch.equal(q.sums.view(-1), z.sum(1).to(torch.int32))
    scales = q.scales.view(-1)
    assert torch.equal(scales[valid], a[valid]) and torch.isnan(scales[~valid]).all()
    assert f.item() == (1 if flagged else 0) == int((~valid).any())


@pytest.mark.parametrize("exponent", [-73, -3, 105])
def test_every_mantissa_of_the_peak(exponent):
    gen = torch.Generator(device="cuda").manual_seed(exponent + 200)
    for chunk in range(8):
        i = torch.arange(chunk << 20, (chunk + 1) << 20, device="cuda", dtype=torch.int32)
        peak = (i | (127 + exponent) << 23).view(torch.float32)
        x = (torch.rand((1 << 20, 32), device="cuda", generator=gen) * 2 - 1) * peak[:, None]
        x[:, 5] = peak * torch.where(i % 2 == 0, 1.0, -1.0)
        x[:, 6] = peak * 0.5  # a tie for many scales
        check(x.view(1024, 32768), False)


def test_outside_the_fast_range():
    gen = torch.Generator(device="cuda").manual_seed(1)
    for scale in (2.0 ** -140, 2.0 ** -100, 2.0 ** -74, 2.0 ** 107, 2.0 ** 126):
        x = torch.randn((4, 4096), device="cuda", generator=gen) * scale
        x[1, :64] = 0.0
        x[2] = x[2].sign() * 2.0 ** -149 if scale < 2.0 ** -139 else x[2]  # peaks that divide to zero are refused
        check(x.clamp(-3e38, 3e38), scale < 2.0 ** -139)
    mixed = torch.randn((4, 4096), device="cuda", generator=gen)
    mixed[0, 40], mixed[1, 100], mixed[2, 4095] = float("inf"), float("nan"), float("-inf")
    check(mixed, True)
    check((mixed.nan_to_num(0, 0, 0) * 1e-42), False)
