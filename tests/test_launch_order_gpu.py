"""Launches are placed beside the end of the kernel before them without being asked to: what that kernel writes (weights,
activations) is still read only when it has ended, eagerly, in a replayed graph and behind a join of two captured streams."""
import pytest
import torch

from qw38_b200 import _lib as L
from qw38_b200 import synth
from qw38_b200.q4k_q8 import (DecodeMmvDesc, PrefillWeight, decode_workspace, launch_decode_mmv, new_q8_input, pack_q8, prefill_project,
                              q4k_q8_project)

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m", [1, 2, 5, 13, 17, 64, 130])
@pytest.mark.parametrize("aligned", [True, False])
def test_weights_and_inputs_written_directly_before(m, aligned):
    n, k = 2048, 2560
    versions = [synth.device_weight(n, k, seed=s) for s in (1, 2)]
    off = 0 if aligned else 4  # unaligned weights take the kernels without bulk copies
    codes, scales = (torch.zeros(t.numel() + 16, dtype=torch.uint8, device=DEV)[off:off + t.numel()] for t in (versions[0].codes, versions[0].scales))
    w = PrefillWeight(codes, scales, n, k)
    g = torch.Generator(device=DEV).manual_seed(m)
    xs = [torch.randn((m, k), device=DEV, generator=g).to(torch.bfloat16) for _ in versions]
    x, f = torch.zeros_like(xs[0]), torch.zeros(1, dtype=torch.int32, device=DEV)
    q, ws = new_q8_input(m, k), decode_workspace(m, n, k)
    outs = [[torch.empty((m, n), device=DEV) for _ in range(2)] for _ in versions]
    entry = launch_decode_mmv if m <= 16 else prefill_project

    def step(sync, side=None):
        for v, src, (o0, o1) in zip(versions, xs, outs):
            for _ in range(3):  # a long predecessor: the last writes come late
                if side is not None:
                    side.wait_stream(torch.cuda.current_stream())
                    with torch.cuda.stream(side):
                        scales.copy_(v.scales)
                else:
                    scales.copy_(v.scales)
                x.copy_(src)
                codes.copy_(v.codes)
                if side is not None:
                    torch.cuda.current_stream().wait_stream(side)
                sync()
                entry(DecodeMmvDesc(w, x, o0, L.EPILOGUE_STORE_FP32), ws, f)
                codes.zero_()
                codes.copy_(v.codes)
                sync()
                pack_q8(x, f, out=q)
                q4k_q8_project(w, q, out=o1)
                codes.zero_()

    def results(run):
        for pair in outs:
            for o in pair:
                o.fill_(-3.0)
        run()
        torch.cuda.synchronize()
        return [o.clone() for pair in outs for o in pair]

    want = results(lambda: step(torch.cuda.synchronize))
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    runs = [lambda: step(lambda: None)]
    for joined in (False, True):
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            step(lambda: None, side if joined else None)
        runs.append(graph.replay)
    for run in runs:
        for _ in range(3):
            assert all(torch.equal(a, b) for a, b in zip(results(run), want))
    assert f.item() == 0
