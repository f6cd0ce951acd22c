"""The fitter's order of roundings: every block against a float32 restatement of the search (one rounding per operation, sums
in index order, candidates in ascending order), over weight distributions that accept few and many candidates."""
import numpy as np
import pytest
import torch

from qw38_b200.q4k_q8 import quantize_q4k_blocks

F = np.float32


def levels(v):
    """Round to nearest even through the 1.5 * 2^23 bias, then clamp to [0, 15]."""
    bits = (v.astype(F) + F(12582912)).astype(F).view(np.uint32)
    return np.clip((bits & 0x7fffff).astype(np.int64) - 0x400000, 0, 15)


def in_order(terms):
    s = terms[:, 0].copy()
    for i in range(1, 32):
        s = (s + terms[:, i]).astype(F)
    return s


def fit_groups(x):
    """[groups, 32] float32 -> step, negated minimum, and the levels of the accepted grid."""
    avg = np.sqrt(in_order(x * x) / F(32)).astype(F)
    w = (avg[:, None] + np.abs(x)).astype(F)
    lo, hi = np.minimum(x.min(1), F(0)), x.max(1)
    sum_w, sum_x = in_order(w), in_order(w * x)
    with np.errstate(all="ignore"):
        grid = F(15) / (hi - lo)
        scale = F(1) / grid

        def error(l, step, base):
            d = (step[:, None] * l).astype(F) + base[:, None] - x
            return in_order(w * (d * d))

        kept = levels(grid[:, None] * (x - lo[:, None])).astype(F)
        best, floor = error(kept, scale, lo), lo.copy()
        for step in range(21):
            g = ((F(-1) + F(0.1) * F(step)) + F(15)) / (hi - floor)
            l = levels(g[:, None] * (x - floor[:, None])).astype(F)
            wl = w * l
            sl, sl2, sxl = in_order(wl), in_order(wl * l), in_order(wl * x)
            det = sum_w * sl2 - sl * sl
            cs, cm = (sum_w * sxl - sum_x * sl) / det, (sl2 * sum_x - sl * sxl) / det
            above = cm > 0
            cs, cm = np.where(above, sxl / sl2, cs), np.where(above, F(0), cm)
            e = error(l, cs, cm)
            take = (det > 0) & (e < best)
            best, scale, floor = np.where(take, e, best), np.where(take, cs, scale), np.where(take, cm, floor)
            kept = np.where(take[:, None], l, kept)
    flat = hi == lo
    return np.where(flat, F(0), scale), np.where(flat, -lo, -floor), np.where(flat[:, None], F(0), kept)


def fit_blocks(x):
    """[blocks, 256] -> codes, and per group the six-bit scale and minimum, d and dmin as fp16."""
    b = len(x)
    scale, low, kept = (v.reshape(b, 8, -1) for v in fit_groups(x.reshape(-1, 32)))
    scale, low = scale[..., 0], low[..., 0]
    with np.errstate(all="ignore"):
        top, top_min = np.maximum(scale.max(1), F(0)), np.maximum(low.max(1), F(0))
        inv = [np.where(t > 0, F(63) / t, F(0)) for t in (top, top_min)]
        d, dmin = (top / F(63)).astype(np.float16), (top_min / F(63)).astype(np.float16)
        six = [np.minimum(63, ((v * i[:, None] + F(12582912)).astype(F).view(np.uint32) & 0x7fffff).astype(np.int64) - 0x400000 & 255)
               for v, i in ((scale, inv[0]), (low, inv[1]))]
        step, off = d.astype(F)[:, None] * six[0].astype(F), dmin.astype(F)[:, None] * six[1].astype(F)
        again = levels((x.reshape(b, 8, 32) + off[..., None]) / step[..., None])
    codes = np.where(step[..., None] != 0, again, kept.astype(np.int64))
    return codes.reshape(b, 256).astype(np.int8), six[0], six[1], d, dmin


def test_restatement_matches_the_committed_vectors(golden):
    codes, _, _, d, dmin = fit_blocks(golden["b_weights"].reshape(-1, 256))
    assert np.array_equal(codes, golden["b_fit_codes"].reshape(-1, 256))
    meta = golden["b_fit_meta"].reshape(-1, 16)
    assert np.array_equal(d.view(np.uint16), meta[:, 0:2].copy().view(np.uint16)[:, 0])
    assert np.array_equal(dmin.view(np.uint16), meta[:, 2:4].copy().view(np.uint16)[:, 0])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["normal", "heavy", "positive", "offset", "coarse", "outlier"])
def test_every_block_equals_the_restatement(kind):
    g = np.random.default_rng(7).standard_normal((6000, 256)).astype(F)
    x = {"normal": g * F(0.02), "heavy": g ** 3, "positive": np.abs(g) + F(3), "offset": g * F(1e-3) - F(1),
         "coarse": np.round(g * 2) / F(8), "outlier": np.where(np.abs(g) > 2.5, g * F(40), g * F(0.01))}[kind].astype(F)
    codes, meta, status = quantize_q4k_blocks(torch.from_numpy(x).to("cuda"), check=False)
    want, sc, mn, d, dmin = fit_blocks(x)
    m = meta.cpu().numpy()
    assert not status.cpu().numpy().any() and np.array_equal(codes.cpu().numpy(), want)
    assert np.array_equal(m[:, 0:2].copy().view(np.uint16)[:, 0], d.view(np.uint16))
    assert np.array_equal(m[:, 2:4].copy().view(np.uint16)[:, 0], dmin.view(np.uint16))
    assert np.array_equal(m[:, 4:8] & 63, sc[:, :4]) and np.array_equal(m[:, 8:12] & 63, mn[:, :4])
