"""Performance cases of the Q4_K x Q8 engine: what a serving process and a model loader have it do.

A case is one pass through the public entry points with everything a program keeps between passes (weights, workspaces,
output buffers, captured graphs) already in hand.  Shapes are those of the benchmark configurations and the tests (hidden
5120, feed-forward 17408, QKV 7168, gate+up 34816); `draw` spreads over the ranges around them, odd sizes included."""
from __future__ import annotations

import math

import torch

from qw38_b200 import _lib as L
from qw38_b200 import (PrefillWeight, dequantize_bf16, launch_overlap, new_q8_input, pack_q8, q4k_q8_mlp, q4k_q8_project,
                       q4k_q8_project_ragged, q8_mlp_workspace_bytes, quantize_q4k_weight, repack_blocks144,
                       set_launch_overlap)
from qw38_b200.q4k_q8 import (DecodeMmvDesc, decode_workspace, launch_decode_mmv, launch_decode_mmv_ranges,
                              prefill_paired_swiglu, prefill_project, reserve_scratch)

DEV = "cuda"
HIDDEN, FFN = 5120, 17408
EPS = 1e-6


def listed():
    return [
        # One token through one attention output projection, residual added: the smallest call of a decode step.
        {"name": "mmv_m1", "kind": "mmv", "m": 1, "n": 5120, "k": 5120},
        # fp32 activations quantised and multiplied for one token: the single-GEMV configuration.
        {"name": "project_f32_m1", "kind": "project", "m": 1, "n": 17408, "k": 5120, "f32": True},
        # A decode layer for four sequences, eager calls: Q/K/V ranges, output projection, MLP chain.
        {"name": "layer_m4", "kind": "layer", "m": 4, "hidden": HIDDEN, "ffn": FFN, "kv": 1024},
        # The MLP chain for an odd decode batch.
        {"name": "mlp_m13", "kind": "mlp", "m": 13, "hidden": HIDDEN, "ffn": FFN},
        # Whole-model decode as servers run it: layers captured in a graph, one token.
        {"name": "stream_m1", "kind": "stream", "m": 1, "layers": 8, "hidden": HIDDEN, "ffn": FFN},
        # The same for a batch of 64 sequences.
        {"name": "stream_m64", "kind": "stream", "m": 64, "layers": 8, "hidden": HIDDEN, "ffn": FFN},
        # The MLP chain over a short prompt chunk of a ragged length.
        {"name": "mlp_m237", "kind": "mlp", "m": 237, "hidden": HIDDEN, "ffn": FFN},
        # Continuous batch: 48 decode rows and prefill chunks of 512, 237 and 1024 tokens through gate+up.
        {"name": "ragged_m1821", "kind": "ragged", "decode": 48, "chunk": 1024, "n": 34816, "k": 5120},
        # A prompt chunk through the prefill engine: gate/up with SwiGLU, then down with the residual.
        {"name": "prefill_m2048", "kind": "prefill", "m": 2048, "hidden": HIDDEN, "ffn": FFN},
        # A long prompt through one projection: the largest call.
        {"name": "project_m8192", "kind": "project", "m": 8192, "n": 17408, "k": 5120, "f32": False},
        # Encoding: fitting a bf16 checkpoint matrix to Q4_K.
        {"name": "fit_bf16", "kind": "fit", "n": 5120, "k": 17408},
        # Loading: native 144-byte blocks to the resident layout, and decoding that to bf16.
        {"name": "layout", "kind": "layout", "n": 17408, "k": 5120},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tile(rng, lo, hi):
    """A multiple of 256 (the super-block length), spread over the logarithm."""
    return max(lo, min(hi, (_log(rng, lo, hi) + 128) // 256 * 256))


def draw(rng):
    kind = rng.choice(["mmv", "project", "project", "layer", "mlp", "mlp", "stream", "ragged", "prefill", "fit", "layout"])
    if kind == "mmv":
        return {"kind": kind, "m": rng.randint(1, 16), "n": _log(rng, 512, 34816), "k": _log(rng, 512, 17408)}
    if kind == "project":
        return {"kind": kind, "m": _log(rng, 1, 8192), "n": _log(rng, 512, 17408), "k": _log(rng, 512, 5120),
                "f32": rng.random() < 0.3}
    if kind == "layer":
        return {"kind": kind, "m": rng.randint(1, 16), "hidden": _tile(rng, 1024, 6144), "ffn": _tile(rng, 2048, 17408),
                "kv": rng.randrange(128, 1025, 8)}
    if kind == "mlp":
        return {"kind": kind, "m": _log(rng, 1, 1024), "hidden": _tile(rng, 512, 5120), "ffn": _tile(rng, 1024, 17408)}
    if kind == "stream":
        return {"kind": kind, "m": _log(rng, 1, 128), "layers": rng.randint(2, 8), "hidden": _tile(rng, 1024, 5120),
                "ffn": _tile(rng, 2048, 17408)}
    if kind == "ragged":
        return {"kind": kind, "decode": rng.randint(1, 64), "chunk": _log(rng, 16, 1024), "n": _log(rng, 1024, 34816),
                "k": _log(rng, 512, 5120)}
    if kind == "prefill":
        return {"kind": kind, "m": _log(rng, 32, 2048), "hidden": _tile(rng, 512, 5120), "ffn": _tile(rng, 1024, 17408)}
    return {"kind": kind, "n": _log(rng, 256, 17408), "k": _tile(rng, 512, 5120)}


def _offsets(case):
    """Row offsets of a ragged batch: single decode rows, then three prefill chunks."""
    c = case["chunk"]
    offs = list(range(case["decode"] + 1))
    for rows in ((c + 1) // 2, max(1, c * 237 // 1024), c):
        offs.append(offs[-1] + rows)
    return offs


# ---- inputs ------------------------------------------------------------------------------------------------------------
class _Inputs:
    """Seeded device tensors with the value distributions of the benchmark configurations."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)

    def bytes(self, *shape):
        return torch.randint(0, 256, shape, dtype=torch.uint8, device=DEV, generator=self.g)

    def normal(self, *shape):
        return torch.randn(shape, device=DEV, generator=self.g)

    def metadata(self, rows):
        """fp16 d and dmin = |N(0,1)| * 2e-3 and twelve bytes of uniform six-bit scales and mins."""
        meta = self.bytes(rows, 16)
        meta[:, :4] = (self.normal(rows, 2).abs() * 2e-3).to(torch.float16).view(torch.uint8)
        return meta

    def weight(self, n, k):
        """Uniform 4-bit codes in split tiles; padded rows and columns hold zeros."""
        groups, tiles = (n + 7) // 8, (k + 255) // 256
        codes = self.bytes(groups, tiles, 8, 128)
        meta = self.metadata(groups * tiles * 8).view(groups, tiles, 8, 16)
        if n % 8:
            codes[-1, :, n % 8:] = 0
            meta[-1, :, n % 8:] = 0
        if k % 256:
            codes[:, -1, :, (k % 256 + 1) // 2:] = 0
            if k % 2:
                codes[:, -1, :, k % 256 // 2] &= 15
        return PrefillWeight(codes.view(-1), meta.view(-1), n, k)

    def activations(self, m, k):
        """Decode rows are N(0,1); prompt rows N(0,1) * 0.5 with one channel in a hundred twenty times larger."""
        x = self.normal(m, k)
        if m > 16:
            x *= 0.5
            x[:, torch.randperm(k, device=DEV, generator=self.g)[:max(1, k // 100)]] *= 20.0
        return x

    def hidden(self, m, width):
        """A residual stream and the RMS gain of its norm."""
        return self.normal(m, width) * 2.0, (self.normal(width) * 0.1).to(torch.bfloat16)


def _flag():
    return torch.zeros(1, dtype=torch.int32, device=DEV)


def _empty(m, n, dtype=torch.float32):
    return torch.empty((m, n), dtype=dtype, device=DEV)


def _bytes(count):
    return torch.empty(count, dtype=torch.uint8, device=DEV)


def _set(hidden, ffn):
    """One layer's projection set: QKV, O, gate+up as one matrix, down."""
    return [(hidden + 2048, hidden), (hidden, hidden), (2 * ffn, hidden), (hidden, ffn)]


def prepare(case, seed):
    r, kind = _Inputs(seed), case["kind"]
    s = {"kind": kind}
    if kind in ("fit", "layout"):
        n, k = case["n"], case["k"]
        if kind == "fit":
            s["weights"] = (r.normal(n, k) * 0.02).to(torch.bfloat16)
        else:
            blocks = r.bytes(n * (k // 256), 144)
            blocks[:, :16] = r.metadata(n * (k // 256))
            s.update(blocks=blocks.view(-1), n=n, k=k)
        return s
    s["failure"] = _flag()
    if kind == "mmv":
        m, n, k = case["m"], case["n"], case["k"]
        x, res = r.activations(m, k).to(torch.bfloat16), r.normal(m, n)
        s.update(desc=DecodeMmvDesc(r.weight(n, k), x, _empty(m, n), L.EPILOGUE_RESIDUAL_ADD_FP32, res),
                 workspace=decode_workspace(m, n, k))
    elif kind == "project":
        m, n, k = case["m"], case["n"], case["k"]
        x = r.activations(m, k)
        s.update(weight=r.weight(n, k), x=x if case["f32"] else x.to(torch.bfloat16), q8=new_q8_input(m, k), out=_empty(m, n))
    elif kind == "ragged":
        offs, n, k = _offsets(case), case["n"], case["k"]
        m = offs[-1]
        s.update(weight=r.weight(n, k), x=r.activations(m, k).to(torch.bfloat16), q8=new_q8_input(m, k), out=_empty(m, n), offsets=offs)
    elif kind == "mlp":
        _prepare_mlp(s, r, case["m"], case["hidden"], case["ffn"])
    elif kind == "layer":
        m, h, kv = case["m"], case["hidden"], case["kv"]
        x, attn = r.activations(m, h).to(torch.bfloat16), r.activations(m, h).to(torch.bfloat16)
        s["ranges"] = [DecodeMmvDesc(r.weight(n, h), x, _empty(m, n, torch.bfloat16)) for n in (h, kv, kv)]
        s["qkv_workspace"] = decode_workspace(m, h + 2 * kv, h)
        _prepare_mlp(s, r, m, h, case["ffn"])
        # the output projection updates the residual stream that the MLP then reads
        s["stream"] = r.normal(m, h) * 2.0
        s["o"] = DecodeMmvDesc(r.weight(h, h), attn, s["residual"], L.EPILOGUE_RESIDUAL_ADD_FP32, s["stream"])
        s["o_workspace"] = decode_workspace(m, h, h)
    elif kind == "prefill":
        m, h, f = case["m"], case["hidden"], case["ffn"]
        x, res = r.activations(m, h).to(torch.bfloat16), r.normal(m, h)
        swiglu = _empty(m, f, torch.bfloat16)
        s.update(gate=r.weight(f, h), up=r.weight(f, h), x=x, swiglu=swiglu,
                 down=DecodeMmvDesc(r.weight(h, f), swiglu, _empty(m, h), L.EPILOGUE_RESIDUAL_ADD_FP32, res),
                 workspace=_bytes(max(decode_workspace(m, f, h).numel(), decode_workspace(m, h, f).numel())))
    elif kind == "stream":
        _prepare_stream(s, r, case)
    return s


def _prepare_mlp(s, r, m, hidden, ffn):
    residual, gamma = r.hidden(m, hidden)
    s.update(m=m, residual=residual, gamma=gamma, gate=r.weight(ffn, hidden), up=r.weight(ffn, hidden), down=r.weight(hidden, ffn),
             out=_empty(m, hidden), workspace=_bytes(q8_mlp_workspace_bytes(m, hidden, ffn)))


def _prepare_stream(s, r, case):
    """Layers of the projection set captured once with overlapped launches: both activation packs of a layer first, so that
    no projection's input is the work of the launch before it."""
    m, hidden, ffn = case["m"], case["hidden"], case["ffn"]
    shapes = _set(hidden, ffn)
    layers = [[r.weight(n, k) for n, k in shapes] for _ in range(case["layers"])]
    x = {k: r.normal(m, k).to(torch.bfloat16) for k in (hidden, ffn)}
    q8 = {k: new_q8_input(m, k) for k in x}
    outs = [[_empty(m, n) for n, _ in shapes] for _ in layers]

    def step():
        for weights, out in zip(layers, outs):
            for k in x:
                pack_q8(x[k], s["failure"], out=q8[k])
            for w, o in zip(weights, out):
                q4k_q8_project(w, q8[w.k], out=o, trusted=True, input_settled=True)

    before = launch_overlap()
    reserve_scratch(16 * m * max(n for n, _ in shapes) * 4)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    set_launch_overlap(True)
    try:
        with torch.cuda.stream(stream):
            step()
            graph = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                step()
    finally:
        set_launch_overlap(before)
    s.update(graph=graph, stream=stream, layers=layers, x=x, q8=q8, outs=outs)


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "fit":
        w = quantize_q4k_weight(s["weights"])
        return w.codes, w.scales
    if kind == "layout":
        w = repack_blocks144(s["blocks"], s["n"], s["k"])
        return w.codes, w.scales, dequantize_bf16(w)
    failure = s["failure"]
    if kind == "mmv":
        launch_decode_mmv(s["desc"], s["workspace"], failure)
        return s["desc"].output, failure
    if kind in ("project", "ragged"):
        q8 = pack_q8(s["x"], failure, out=s["q8"])
        if kind == "project":
            q4k_q8_project(s["weight"], q8, out=s["out"])
        else:
            q4k_q8_project_ragged(s["weight"], q8, s["offsets"], out=s["out"])
        return s["out"], q8.codes, q8.scales, q8.sums, failure
    if kind == "mlp":
        return _run_mlp(s), failure
    if kind == "layer":
        launch_decode_mmv_ranges(s["ranges"], s["qkv_workspace"], failure)
        launch_decode_mmv(s["o"], s["o_workspace"], failure)
        return [d.output for d in s["ranges"]], s["residual"], _run_mlp(s), failure
    if kind == "prefill":
        prefill_paired_swiglu(s["gate"], s["up"], s["x"], s["swiglu"], s["workspace"], failure)
        prefill_project(s["down"], s["workspace"], failure)
        return s["swiglu"], s["down"].output, failure
    s["graph"].replay()
    return s["outs"], failure


def _run_mlp(s):
    q4k_q8_mlp(s["gate"], s["up"], s["down"], s["residual"], s["gamma"], EPS, s["out"], s["m"], s["workspace"],
               pending_failure=s["failure"])
    return s["out"]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def _weight_bytes(n, k):
    return (n + 7) // 8 * 8 * ((k + 255) // 256) * 144


def _q8_bytes(m, k):
    pk = (k + 255) // 256 * 256
    return m * (pk + pk // 32 * 8)


def _mlp_work(m, hidden, ffn):
    """The chain: residual in, gain, three matrices, result out; what lies between can stay on the chip."""
    return 3 * _weight_bytes(ffn, hidden) + 2 * m * hidden * 4 + hidden * 2, 6 * m * hidden * ffn


def work(case):
    kind, m = case["kind"], case.get("m", 0)
    if kind == "fit":  # 21 candidate grids and the first, each a pass over the weights with about 17 operations per weight
        n, k = case["n"], case["k"]
        return {"bytes": n * k * 2 + _weight_bytes(n, k), "flops": n * k * 22 * 17}
    if kind == "layout":
        n, k = case["n"], case["k"]
        return {"bytes": n * (k // 256) * 144 + _weight_bytes(n, k) + n * k * 2, "flops": 0}
    if kind == "mmv":
        n, k = case["n"], case["k"]
        return {"bytes": _weight_bytes(n, k) + m * k * 2 + 2 * m * n * 4, "flops": 2 * m * n * k}
    if kind in ("project", "ragged"):
        n, k = case["n"], case["k"]
        if kind == "ragged":
            m = _offsets(case)[-1]
        x = m * k * (4 if case.get("f32") else 2)
        return {"bytes": _weight_bytes(n, k) + x + _q8_bytes(m, k) + m * n * 4, "flops": 2 * m * n * k}
    h, f = case["hidden"], case["ffn"]
    if kind == "prefill":
        return {"bytes": 3 * _weight_bytes(f, h) + m * h * 2 + m * f * 2 + 2 * m * h * 4, "flops": 6 * m * h * f}
    if kind == "stream":
        one = sum(_weight_bytes(n, k) + m * n * 4 for n, k in _set(h, f)) + m * (h + f) * 2
        return {"bytes": case["layers"] * one, "flops": case["layers"] * sum(2 * m * n * k for n, k in _set(h, f))}
    b, fl = _mlp_work(m, h, f)
    if kind == "layer":
        kv = case["kv"]
        b += _weight_bytes(h, h) + 2 * m * h * 2 + 2 * m * h * 4 + sum(_weight_bytes(n, h) + m * n * 2 for n in (h, kv, kv))
        fl += 2 * m * h * (2 * h + 2 * kv)
    return {"bytes": b, "flops": fl}


def tolerance(case):
    kind = case["kind"]
    if kind in ("fit", "layout"):
        return "exact"
    if kind in ("mlp", "layer", "prefill"):
        # a bf16 rounding of the SwiGLU product that lands on the other side of a tie moves one activation code
        return {"rel": 2e-3}
    return {"rel": 1e-5}  # fp32 sums in another order; codes and flags are whole numbers and stay the same
