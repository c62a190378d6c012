"""Decode steps of the one-launch attention kernel (csrc/attention_bias.cu, attn_step_kernel) where its parts carry something from one turn to the next:
several passes of a CTA's 128 keys with scores that grow or fall along the sequence, clusters of 8, 4, 2 and 1 and more units than SMs, cache
capacities on both sides of the line to the tiled kernel, gated outputs in both formats, and operands that are not finite. The slots hold prefixes of
one sequence, so that one run of the plain oracle gives the logits of all of them."""
import numpy as np
import pytest
import torch

import test_infinite_operands_gpu as INF
import test_katadra_gpu as KA
import test_kuvelix_gpu as KV
import test_sofopel_gpu as SO

pytestmark = pytest.mark.gpu

# Logits of true fp32: projections, scores, output, feed-forward-free residual and head are sums of at most 256 fp32 terms, about 2^-24 sqrt(256 / 2) = 7e-7 of
# their result each (2-norm), and so is the weighted mean of the values (a warp's share of 2400 keys, then 16 warps, then 8 CTAs): five in a row.
# A row of 150 logits may be off by three times the rms of all rows.
F32 = 3 * 5 * 7e-7


def worst(got, ref):
    e = (got.double().cpu() - ref).pow(2).mean(-1).sqrt() / ref.std(-1)
    return float(e.max())


def decode(mod, cfg, w, toks, lengths, dtype=torch.float32, steps=2, capacity=None):
    """Logits [slot, step, vocab] of the engine, and the oracle's"""
    n = max(lengths) + steps
    model, _ = mod.build(cfg, dtype, weights=w, max_batch=len(lengths), max_seq=capacity or n, max_rows=min(n, 2400))
    eng = model._ensure_engine()
    kv = eng.new_kv(len(lengths), capacity or n)
    for b, at in enumerate(lengths):
        eng.append_tokens(kv, b, toks[:at], restart=True)
    got = torch.stack([eng.decode_step(kv, torch.tensor([toks[at + t] for at in lengths], dtype=torch.int32)).clone() for t in range(steps)], 1).cpu()
    model.invalidate_engine()
    out = mod.O.forward(cfg, w, toks[:n])
    ref = torch.as_tensor(np.asarray(out), dtype=torch.float64)
    return got, torch.stack([ref[at:at + steps] for at in lengths])


def rising(heads, kv, dim, vdim, n, order, seed=0):
    """A prompt along which every query's scores rise (or fall) by some 20: entry 0 of the stream goes with the token, entry 1 is the same for all"""
    cfg = KV.config([KV.layer(KV.attn(heads, kv, dim, vdim, 0, scale=0.2), None)])
    w = KV.O.random_weights(cfg, seed=seed)
    e, k, q = w["embed"].copy(), w["l0.mix.k"].copy(), w["l0.mix.q"].copy()
    e[:, 0], e[:, 1] = np.arange(cfg["vocab"]) / 64.0, 1.0
    k[::dim], q[::dim] = 0, 0
    k[::dim, 0], q[::dim, 1] = 4.0, 4.0
    w["embed"], w["l0.mix.k"], w["l0.mix.q"] = KV.O.bf16_round(e), k, q
    toks = [p * cfg["vocab"] // n for p in range(n)]
    return cfg, w, toks if order == "rising" else toks[::-1]


@pytest.mark.parametrize("order", ["rising", "falling"])
@pytest.mark.parametrize("heads,kv,dim,vdim", [(1, 1, 32, 32), (4, 2, 64, 100), (3, 1, 96, 64), (4, 1, 128, 128), (6, 1, 32, 36), (16, 8, 32, 128)])
def test_running_maximum_over_many_passes(heads, kv, dim, vdim, order):
    cfg, w, toks = rising(heads, kv, dim, vdim, 2402, order)
    got, ref = decode(KV, cfg, w, toks, [2400, 1025, 129, 128])
    assert worst(got, ref) < F32


@pytest.mark.parametrize("slots,kv,heads,vdim", [(4, 8, 8, 32), (8, 8, 8, 36), (10, 8, 16, 32), (20, 8, 32, 32), (40, 2, 10, 4), (20, 2, 4, 128)])
def test_clusters_of_every_size(slots, kv, heads, vdim):
    """32, 64 units (clusters of 4 and 2), 80, 160, 160 and 40 of them"""
    cfg = KV.config([KV.layer(KV.attn(heads, kv, 32, vdim, 8, scale=0.2), None)])
    w = KV.O.random_weights(cfg, seed=slots)
    lengths = [1 + (b * 299) // (slots - 1) for b in range(slots)]
    got, ref = decode(KV, cfg, w, KV.tokens_for(cfg, 302), lengths)
    assert worst(got, ref) < F32


@pytest.mark.parametrize("size,keep", [(1500, 70), (130, 5), (40, 700), (2000, 0)])
@pytest.mark.parametrize("heads,kv", [(4, 2), (8, 2)])
def test_windows_and_kept_positions_over_many_passes(heads, kv, size, keep):
    cfg = SO.config([SO.layer(SO.win(heads, kv, 64, 64, size, keep, 16, scale=0.6), None)])
    w = SO.O.random_weights(cfg, seed=size)
    got, ref = decode(SO, cfg, w, SO.tokens_for(cfg, 2302), [2300, 1999, 1500, 699])
    assert worst(got, ref) < F32


def biased(heads, kv, rel=None):
    left = {"heads": heads, "kv_heads": kv, "dim": 32, "vdim": 64, "bias_max": 64, "scale": 0.3, "softcap": 5.0, "q_temp": {"coef": 0.5, "every": 16}, "rel_rows": 16}
    cfg = KA.config([{"type": "parallel", "mlp": None, "mixer": {"left": left, "right": {"heads": 1, "dim": 8, "decay_rank": 2}, "left_scale": 1.0, "right_scale": 0.5}}], width=72)
    w = KA.O.random_weights(cfg, seed=heads)
    if rel is not None:
        w["l0.mix.left.rel"] = rel(w["l0.mix.left.rel"].clone())
    return cfg, w


@pytest.mark.parametrize("heads", [4, 6, 2])
def test_biases_and_soft_caps_over_many_passes(heads):
    """20 slots of 2 key/value heads: 40 units and more, so 350 or 700 keys a CTA. The bias falls by some 10 with the distance, and rises."""
    for sign in (1.0, -1.0):
        cfg, w = biased(heads, 2, lambda r: (r + sign * torch.linspace(5, -5, len(r))[:, None]).bfloat16().to(r.dtype))
        lengths = [700 - 31 * b for b in range(20)]
        got, ref = decode(KA, cfg, w, KA.tokens_for(cfg, 702), lengths)
        assert worst(got, ref) < F32


def test_both_sides_of_the_line_to_the_tiled_kernel():
    """One slot, one head, 8 CTAs: capacities of up to 8192 positions stay in one launch. Close to the oracle on both sides, by two kernels."""
    cfg = SO.config([SO.layer(SO.win(1, 1, 32, 32, None, None, 8), None)])
    w = SO.O.random_weights(cfg, seed=2)
    toks = SO.tokens_for(cfg, 900)
    a, ref = decode(SO, cfg, w, toks, [898], capacity=8192)
    b, _ = decode(SO, cfg, w, toks, [898], capacity=8193)
    assert worst(a, ref) < F32 and worst(b, ref) < F32 and not torch.equal(a, b)


@pytest.mark.parametrize("slots", [1, 3, 20])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_channel_gates_in_both_formats(slots, dtype, monkeypatch):
    """20 requests in bf16: the attention writes the next product's operand. bf16: against the FMA kernels, which take it in fp32 and round it themselves"""
    cfg = KV.config([KV.layer(KV.attn(6, 2, 64, 128, 16, scale=0.15), None)])
    w = KV.O.random_weights(cfg, seed=7)
    toks, lengths = KV.tokens_for(cfg, 302), [300 - 13 * b for b in range(slots)]
    got, ref = decode(KV, cfg, w, toks, lengths, dtype)
    if dtype == torch.float32:
        assert worst(got, ref) < F32
        return
    monkeypatch.setenv("B2_SEQ_TC", "0")
    plain, _ = decode(KV, cfg, w, toks, lengths, dtype)
    # against 64 bits: operands rounded to bf16 four times in a row (2^-9 of each entry, rms 0.6 of that), three times the rms for one row; against
    # each other: now and then an entry falls on the other side of such a rounding
    assert worst(got, ref) < 3 * 4 * 0.6 * 2 ** -9 and worst(got, plain.double()) < 2 ** -9


INFTY = float("inf")


@pytest.mark.parametrize("slots", [1, 20])
@pytest.mark.parametrize("name,rel", [
    ("only_itself", lambda r: torch.where(torch.arange(len(r))[:, None] > 0, torch.full_like(r, -INFTY), r)),
    ("nothing_near", lambda r: torch.where(torch.arange(len(r))[:, None] < 5, torch.full_like(r, -INFTY), r)),
    ("nothing", lambda r: torch.full_like(r, -INFTY)),
    ("plus", lambda r: torch.where(torch.arange(len(r))[:, None] == 9, torch.full_like(r, INFTY), r)),
    ("nan", lambda r: torch.where(torch.arange(len(r))[:, None] == 9, torch.full_like(r, float("nan")), r))])
def test_biases_that_are_not_finite(name, rel, slots):
    """Scores of minus infinity weigh nothing, also where whole passes, warps and CTAs have no others; a row without any, or with a score that is not a
    number or plus infinity, is NaN."""
    cfg, w = biased(4, 2, rel)
    lengths = [700 - 31 * b for b in range(slots)]
    got, ref = decode(KA, cfg, w, KA.tokens_for(cfg, 702), lengths)
    bad = ref.isnan().any(-1)
    assert torch.equal(got.isnan().any(-1), bad) and bool(bad.any()) == (name in ("nothing", "plus", "nan"))
    if not bad.all():
        assert worst(got[~bad], ref[~bad]) < F32


@pytest.mark.parametrize("chunk", [None, 25])
def test_a_key_with_an_infinite_entry(chunk):
    """Every later query looks the other way: the key is as good as absent"""
    cfg = SO.config([dict(SO.diff(2, 1, 64, 72, None, chunk, 0), mlp=None)], width=64, vocab=90, mult=1.0)
    w, toks = INF.special_token(cfg, 5)
    k, q = w["l0.mix.k"].copy(), w["l0.mix.q"].copy()
    k[0], q[0], q[2 * 64] = 0, 0, 0
    k[0, 0], q[0, 1], q[2 * 64, 1] = INF.HUGE, -1, -1
    w["l0.mix.k"], w["l0.mix.q"] = k, q
    got, ref = decode(SO, cfg, w, toks, [22, 23, 24, 40, 88])
    assert bool(ref.isfinite().all()) and worst(got, ref) < F32


@pytest.mark.parametrize("chunk", [None, 25])
def test_an_infinite_value(chunk):
    """Slots that do not see it are as they would be without it; those that do are not finite"""
    cfg = SO.config([dict(SO.diff(2, 1, 64, 72, None, chunk, 0), mlp=None)], width=64, vocab=90, mult=1.0)
    w, toks = INF.special_token(cfg, 6)
    v = w["l0.mix.v"].copy()
    v[1] = 0
    v[1, 0] = INF.HUGE
    w["l0.mix.v"] = v
    lengths = [5, 19, 22, 30, 60, 88]
    got, ref = decode(SO, cfg, w, toks, lengths, steps=1)
    seen = [at >= 21 and (chunk is None or at // chunk == 21 // chunk) for at in lengths]
    for b, s in enumerate(seen):
        assert not got[b].isfinite().all() if s else worst(got[b], ref[b]) < F32
