"""The fp16-plane kernel (automatic choice beyond sixteen tokens): edges of its row, token and K tiles, short and cut tiles,
activation scales far apart, overlapped launches in a replayed graph, and scratch that streams and graphs do not share."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from qw38_b200 import _lib as L
from qw38_b200 import set_launch_overlap, synth
from qw38_b200.q4k_q8 import (DecodeMmvDesc, PrefillWeight, decode_workspace, new_q8_input, pack_q8, prefill_paired_swiglu,
                              prefill_project, q4k_q8_project)
from tests.helpers import assert_close_contract

pytestmark = pytest.mark.gpu
DEV = "cuda"


def flag():
    return torch.zeros(1, dtype=torch.int32, device=DEV)


def kernel_status():
    v = ctypes.c_int(-1)
    assert L.load().q4k_kernel_status(ctypes.byref(v)) == 0
    return v.value


def weight(n, k, seed):
    hc, hs = synth.split_tiles(*synth.logical_q4k(n, k, seed=seed))
    return PrefillWeight.from_host(hc, hs, n, k), hc, hs


@pytest.mark.parametrize("m,n,k", [(1, 256, 256), (16, 9, 512), (17, 1, 256), (32, 257, 259), (33, 136, 768), (64, 640, 1280),
                                   (65, 128, 1024), (97, 1000, 2560), (128, 520, 300), (129, 264, 5120), (224, 2056, 1536),
                                   (64, 72, 17408)])
def test_edges_match_the_oracle(m, n, k):
    w, hc, hs = weight(n, k, seed=m + n)
    x = synth.activations(m, k, seed=k, scale=0.5, outlier_frac=0.01)
    q = pack_q8(torch.from_numpy(x).to(DEV), flag())
    z, a, s, _ = orc.q8_quantize(x)
    ref = orc.project(hc, hs, n, q.padded_k, z, a, s)
    guarded = torch.full((m * n + 2,), -7.0, dtype=torch.float32, device=DEV)
    y = q4k_q8_project(w, q, out=guarded[1:-1].view(m, n), kernel=L.KERNEL_F16)
    assert guarded[0].item() == -7.0 and guarded[-1].item() == -7.0
    assert_close_contract(y.cpu().numpy(), ref)
    res = torch.from_numpy(synth.activations(m, n, seed=5)).to(DEV)
    assert torch.equal(q4k_q8_project(w, q, kernel=L.KERNEL_F16, residual=res), y + res), "residual is the last fp32 add"
    assert kernel_status() == 0


@pytest.mark.parametrize("m", [17, 64, 130])
def test_scales_far_apart(m):
    """A token of 1e30, a super-block 2^40 above the others of its token (they keep powers of two of their own) and one value
    above 2^97: all finite, and accurate relative to each row's size."""
    n, k = 264, 1280
    w, hc, hs = weight(n, k, seed=4)
    x = synth.activations(m, k, seed=11)
    x[0, :] *= 1e30
    x[m // 2, 300:340] *= 1e12
    x[m - 1, 1000] = 2e29
    q = pack_q8(torch.from_numpy(x).to(DEV), flag())
    z, a, s, _ = orc.q8_quantize(x)
    y = q4k_q8_project(w, q).cpu().numpy()
    ref = orc.project(hc, hs, n, k, z, a, s).astype(np.float64)
    rms = np.sqrt((ref ** 2).mean(axis=1, keepdims=True))
    assert np.isfinite(y).all() and (np.abs(y - ref) <= 2e-3 * np.maximum(np.abs(ref), 1e-3 * rms)).all()
    # the super-blocks beside the large one, on their own: the weights of all others are zero
    only = w.codes.clone().view(n // 8, 5, 8, 128)
    mins = w.scales.clone().view(n // 8, 5, 8, 16)
    only[:, 1] = 0
    mins[:, 1] = 0
    y1 = q4k_q8_project(PrefillWeight(only.view(-1), mins.view(-1), n, k), q).cpu().numpy()[m // 2].astype(np.float64)
    r1 = orc.project(only.cpu().numpy().reshape(-1), mins.cpu().numpy().reshape(-1), n, k, z, a, s)[m // 2].astype(np.float64)
    assert np.abs(y1 - r1).max() <= 1e-5 * np.sqrt((r1 ** 2).mean())
    assert kernel_status() == 0


def test_overlapped_graph_and_streams_reproduce_the_serial_result():
    """Chains of projections with settled inputs, whose planes are written beside the projection before them, in a graph
    with overlapped launches; two graphs and eager calls on three streams at once.  All bitwise the serial results."""
    shapes = [(7168, 1280), (640, 5120), (5120, 1280), (1000, 5120)]
    ws = [synth.device_weight(n, k, seed=90 + i) for i, (n, k) in enumerate(shapes)]
    qs = {}
    for m in (64, 40, 130):
        for k in (1280, 5120):
            x = torch.randn((m, k), device=DEV, generator=torch.Generator(device=DEV).manual_seed(m + k))
            qs[(m, k)] = pack_q8(x, flag())

    def outputs():
        return {(m, i): torch.full((m, n), -3.0, device=DEV) for m in (64, 40, 130) for i, (n, _) in enumerate(shapes)}

    def chain(outs, settled):
        for m in (64, 40, 130):
            for i, (_, k) in enumerate(shapes):
                q4k_q8_project(ws[i], qs[(m, k)], out=outs[(m, i)], trusted=True, input_settled=settled)

    want = outputs()
    chain(want, False)
    torch.cuda.synchronize()
    graphs = []
    try:
        set_launch_overlap(True)
        for _ in range(2):
            outs, stream, graph = outputs(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                chain(outs, True)
                chain(outs, True)
            graphs.append((graph, stream, outs))
    finally:
        set_launch_overlap(False)
    eager, side = outputs(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        for graph, stream, _ in graphs:
            with torch.cuda.stream(stream):
                graph.replay()
        with torch.cuda.stream(side):
            chain(eager, False)
    torch.cuda.synchronize()
    for outs in [g[2] for g in graphs] + [eager]:
        for key in want:
            assert torch.equal(outs[key], want[key]), key
    assert kernel_status() == 0


@pytest.mark.parametrize("m,n,k", [(17, 136, 200), (33, 264, 1003), (64, 264, 6400), (130, 520, 2560), (131, 264, 18688), (800, 128, 17408)])
def test_rows_are_quantised_as_the_pack_does(m, n, k):
    """Prefill entries hand the bf16 rows to the kernel's own quantiser: bitwise the pack and the projection, for every number
    of super-blocks per warp, row alignments, several passes, gate and up in one launch, and a value that is not finite."""
    (w, _, _), (w2, _, _) = weight(n, k, seed=m), weight(n, k, seed=m + 1)
    x = torch.from_numpy(synth.activations(m, k, seed=k, scale=0.5, outlier_frac=0.01)).to(DEV).to(torch.bfloat16)
    f, ws = flag(), decode_workspace(m, n, k)
    q = pack_q8(x, f)
    want = [q4k_q8_project(v, q) for v in (w, w2)]
    out = torch.empty((m, n), device=DEV)
    prefill_project(DecodeMmvDesc(w, x, out, L.EPILOGUE_STORE_FP32), ws, f)
    assert torch.equal(out, want[0]) and f.item() == 0
    # input where a first pass would write (the fp32 rows of the workspace): the pack comes first
    at = ws.numel() // 2 * 2 - x.numel() * 2
    inside = ws[at // 16 * 16:at // 16 * 16 + x.numel() * 2].view(torch.bfloat16).view(m, k) if at > m * k * 3 else None
    if inside is not None:
        inside.copy_(x)
        prefill_project(DecodeMmvDesc(w, inside, out, L.EPILOGUE_STORE_FP32), ws, f)
        assert torch.equal(out, want[0])
    both = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
    prefill_paired_swiglu(w, w2, x, both, ws, f)
    ref = torch.nn.functional.silu(want[0].double()) * want[1].double()
    assert (both.double() - ref).abs().max() <= ref.abs().max() * 2.0 ** -8 and f.item() == 0
    x[m - 1, k - 1] = float("nan")
    prefill_project(DecodeMmvDesc(w, x, out, L.EPILOGUE_STORE_FP32), ws, f)
    assert f.item() == 1 and kernel_status() == 0


def test_overlap_switched_inside_a_capture():
    """Projections with settled inputs, launch overlap off and on in turn within one graph: bitwise the serial results."""
    n, k = 5120, 2560
    ws = [synth.device_weight(n, k, seed=60 + i) for i in range(6)]
    q = pack_q8(torch.randn((64, k), device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)), flag())
    want = [q4k_q8_project(w, q) for w in ws]
    outs = [torch.full((64, n), -3.0, device=DEV) for _ in ws]
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        with torch.cuda.graph(graph, stream=stream):
            for i, (w, out) in enumerate(zip(ws * 3, outs * 3)):
                set_launch_overlap(i % 3 != 0)
                q4k_q8_project(w, q, out=out, trusted=True, input_settled=True)
    finally:
        set_launch_overlap(False)
    for _ in range(20):
        for out in outs:
            out.fill_(-3.0)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outs, want))
    assert kernel_status() == 0


def exact(codes, meta, z, a):
    """The equation in 64 bits from logical codes and metadata, on the device."""
    p = meta[..., 4:].astype(np.int64)
    sc = np.concatenate([p[..., 0:4] & 63, (p[..., 8:12] & 15) | (p[..., 0:4] >> 6 << 4)], -1)
    mn = np.concatenate([p[..., 4:8] & 63, (p[..., 8:12] >> 4) | (p[..., 4:8] >> 6 << 4)], -1)
    d, dmin = (np.ascontiguousarray(meta[..., i:i + 2]).view(np.float16).astype(np.float64) for i in (0, 2))
    w = np.repeat((d * sc).reshape(len(codes), -1), 32, 1) * codes - np.repeat((dmin * mn).reshape(len(codes), -1), 32, 1)
    x = z.astype(np.float64) * np.repeat(a.astype(np.float64), 32, 1)
    return (torch.from_numpy(x).to(DEV) @ torch.from_numpy(w).to(DEV).T).cpu().numpy()


# Each super-block: at most sixteen steps of the tensor core at full magnitude, each truncated by up to 2^-23 of the sum so far
# (the mean is compensated, what is left spreads over about 2^-23), then an fp32 addition.  Sums that lose nothing come out
# 2^-22 = 2.4e-7 too large, and the two planes carry x to 2^-23.  Measured, of a token's norm: 2.2e-7 to 3.9e-7 (the int8
# kernel 0.5e-7 to 1.9e-7); 1e-6 is two and a half times that.
@pytest.mark.parametrize("m,n,k", [(17, 264, 512), (64, 520, 5120), (130, 264, 17408)])
@pytest.mark.parametrize("kind", ["dense", "outliers", "one value per super-block", "one value"])
def test_error_against_64_bits(m, n, k, kind):
    codes, meta = synth.logical_q4k(n, k, seed=k)
    hc, hs = synth.split_tiles(codes, meta)
    w = PrefillWeight.from_host(hc, hs, n, k)
    x = synth.activations(m, k, seed=m, scale=0.5, outlier_frac=0.01 if kind == "outliers" else 0.0)
    if kind.startswith("one"):
        keep = np.random.default_rng(m).integers(0, 256, (m, k // 256)) + np.arange(0, k, 256)
        mask = np.zeros_like(x)
        np.put_along_axis(mask, keep if "per" in kind else keep[:, :1], 1.0, 1)
        x = x * mask
    q = pack_q8(torch.from_numpy(x).to(DEV), flag())
    ref = exact(codes, meta, q.codes.cpu().numpy(), q.scales.cpu().numpy())
    norm = np.sqrt((ref ** 2).sum(1))
    for kernel in (L.KERNEL_F16, L.KERNEL_TCGEN05):
        y = q4k_q8_project(w, q, kernel=kernel).cpu().numpy().astype(np.float64)
        err = np.sqrt(((y - ref) ** 2).sum(1)) / norm
        assert err.max() <= 1e-6
    assert kernel_status() == 0
