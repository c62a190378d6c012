"""Linears of 1..16 rows on streamed bf16 weights (csrc/linear_stream.cu) against 64-bit products and against the FMA kernels on the same bf16
operands: one layer of a model, at row counts around the two column tiles of 8, input sizes around the units of 128 that the warps share, and
output sizes that are no multiple of a tile of 16; with biases, activations, sums onto the residual stream and every gated unit."""
import numpy as np
import pytest
import torch

import test_kuvelix_gpu as KV
import test_ramosun_gpu as RA
from oracle import sofopel_oracle as O
from test_sofopel_gpu import config, diff, gla, tokens_for, win

pytestmark = pytest.mark.gpu


def bound(*sizes):
    """Both sides multiply the same bf16 operands and add up in fp32, in other orders (1e-7 of a result). That leaves the operands of the NEXT
    product equal but for the odd entry that falls on the other side of a bf16 rounding: it moves by 2^-8 of itself, and a sum over K entries
    by 2^-8 |entry| / (rms sqrt(K)). Room for one such entry of three times the rms in the smallest of the layer's sums."""
    return 3 * 2 ** -8 / min(sizes) ** 0.5


def sofopel(cfg, w, **limits):
    from llava.model import SofopelConfig, SofopelForCausalLM

    return SofopelForCausalLM(SofopelConfig(**cfg), {k: torch.from_numpy(v).bfloat16() for k, v in w.items()}, dtype=torch.bfloat16, max_batch=2, max_seq=64,
                              max_rows=32, **limits)


def outputs(model, toks, n, slots=1):
    """Residual stream and logits of a prompt of n tokens, then logits of decode steps of `slots` requests"""
    eng = model._ensure_engine()
    kv = eng.new_kv(slots, 64)
    for b in range(slots):
        out = eng.append_tokens(kv, b, toks[:n], list(range(n)), restart=True, residuals=True)
    out = [out[0].flatten().double(), out[1][-1].flatten().double()]
    out += [eng.decode_step(kv, torch.tensor([t] * slots, dtype=torch.int32)).flatten().double() for t in toks[n:]]
    torch.cuda.synchronize()
    model.invalidate_engine()
    return out


def residuals(cfg, w, n, steps):
    return outputs(sofopel(cfg, w), tokens_for(cfg, n + steps), n)


def both_ways(run, monkeypatch, limit):
    """The streamed form and (B2_SEQ_TC=0) the FMA kernels: close, and not the same bits, i.e. two kernels and not one"""
    monkeypatch.setenv("B2_SEQ_TC", "1")
    got = run()
    monkeypatch.setenv("B2_SEQ_TC", "0")
    ref = run()
    for a, b in zip(got, ref):
        assert float((a - b).norm() / b.norm()) <= limit
    assert not all(torch.equal(a, b) for a, b in zip(got, ref))
    assert not all(torch.equal(a, b) for a, b in zip(got[2:], ref[2:]))   # the decode steps by themselves


@pytest.mark.parametrize("width,vocab", [(64, 101), (72, 33), (136, 1003), (264, 50), (1160, 301), (2056, 17)])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16])
def test_head_against_64_bits(width, vocab, n):
    """Logits from the residual stream that the engine returns, normed and rounded to bf16 here. fp32 sums are off by 1e-7 of their terms; an entry
    that falls on the other side of a bf16 rounding moves by up to 2^-7 of itself: room for two such entries of three times the rms."""
    cfg = config([dict(win(1, 1, 8, 8, None, None, 0), mlp=None)], width=width, vocab=vocab)
    w = O.random_weights(cfg, seed=n)
    logits, stream = outputs(sofopel(cfg, w), tokens_for(cfg, n), n)
    x = torch.as_tensor(O.rms_norm(stream.cpu().numpy().reshape(n, width), np.asarray(w["final.norm"], np.float64), float(cfg["norm"]["eps"])))
    head = torch.as_tensor(np.asarray(w["head"], np.float64))
    ref = x.bfloat16().double() @ head.T
    tol = 2 * 2 ** -7 * 3 * x.pow(2).mean(1, keepdim=True).sqrt() * head.abs().max() + 1e-6
    assert bool(((logits.cpu().reshape(n, vocab) - ref).abs() <= tol).all())


@pytest.mark.parametrize("width,ff", [(64, 24), (64, 100), (72, 136), (136, 40), (264, 1032), (1160, 272)])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17])
def test_streamed_weights_equal_the_fma_kernels(width, ff, n, monkeypatch):
    cfg = config([dict(win(5, 1, 24, 40, None, None, 8), mlp={"kind": "dense", "ff": ff, "limit": 7.0})], width=width, vocab=101)
    w = O.random_weights(cfg, seed=3)
    both_ways(lambda: residuals(cfg, w, n, 2), monkeypatch, bound(width, ff, 5 * 40))


SLOTS = [(1, 1), (9, 1), (3, 2), (5, 9), (2, 16)]


# (that feed-forward's norm rides inside the products of fewer than 4 rows, which have a kernel of their own)
@pytest.mark.parametrize("name,n,slots", [(m, *s) for m in ("bounded", "biased") for s in SLOTS] + [("gelu", 9, 4), ("gelu", 5, 9), ("gelu", 4, 16)])
def test_units_biases_and_slots(name, n, slots, monkeypatch):
    """A gated unit whose bounds bite, biased projections with a tanh-GELU unit, a GELU feed-forward; decode steps of 1..16 requests"""
    if name == "bounded":
        cfg = config([dict(win(5, 1, 24, 40, None, None, 8), mlp={"kind": "dense", "ff": 104, "limit": 0.5})], width=136, vocab=101)
        mod, w = None, O.random_weights(cfg, seed=4)
    elif name == "biased":
        mod, cfg = KV, KV.config([KV.layer(KV.attn(4, 1, 24, 40, 12), {"kind": "dense", "ff": 104})], width=136, vocab=101)
    else:
        mod, cfg = RA, RA.config([RA.layer(RA.AT, {"kind": "dense", "ff": 104})], width=136, vocab=101)

    def run():
        toks = tokens_for(cfg, n + 3)
        if mod is not None:
            return outputs(mod.build(cfg, torch.bfloat16, max_batch=slots, max_seq=64, max_rows=32)[0], toks, n, slots)
        from llava.model import SofopelConfig, SofopelForCausalLM

        model = SofopelForCausalLM(SofopelConfig(**cfg), {k: torch.from_numpy(v).bfloat16() for k, v in w.items()}, dtype=torch.bfloat16, max_batch=slots,
                                   max_seq=64, max_rows=32)
        return outputs(model, toks, n, slots)

    both_ways(run, monkeypatch, bound(104, 136, 4 * 24))


# One CTA of 16 warps an SM or two of 8, whichever has the shorter longest chain: tiles that fill both forms' CTAs once, twice and a little more
@pytest.mark.parametrize("width,vocab", [(72, 2376), (264, 2600), (1024, 3001), (1024, 4736), (1032, 4745), (520, 9500), (2048, 2377), (2056, 2600), (4096, 5003)])
@pytest.mark.parametrize("n", [1, 8, 9, 16])
def test_several_tiles_a_block(width, vocab, n):
    test_head_against_64_bits(width, vocab, n)


@pytest.mark.parametrize("width,ff", [(136, 2376), (264, 2504), (1024, 2400), (2048, 1200)])
@pytest.mark.parametrize("n", [1, 8, 9, 16])
def test_several_gated_tiles_a_block(width, ff, n, monkeypatch):
    test_streamed_weights_equal_the_fma_kernels(width, ff, n, monkeypatch)


# A feed-forward whose products run in the launches of the mixer's first and last: tiles of both kinds in a launch, units of two products in a sum
@pytest.mark.parametrize("mixer", ["gla", "diff", "win"])
@pytest.mark.parametrize("width,ff", [(136, 72), (264, 1048), (1160, 272), (2048, 136)])
@pytest.mark.parametrize("n", [1, 3, 4, 8, 9, 16])
def test_products_that_share_a_launch(mixer, width, ff, n, monkeypatch):
    mix = {"gla": gla(3, 16, 40), "diff": diff(4, 2, 16, 24, 3, 13, 8), "win": win(5, 1, 24, 40, 11, 3, 8)}[mixer]
    cfg = config([dict(mix, mlp={"kind": "dense", "ff": ff, "limit": 7.0})], width=width, vocab=101)
    w = O.random_weights(cfg, seed=5)
    both_ways(lambda: residuals(cfg, w, n, 2), monkeypatch, bound(width, ff, 3 * 40, 4 * 24))


# One row normed on its way into the launch of the first products, and into the head: widths around one and several turns of a CTA, the widest and one beyond
@pytest.mark.parametrize("width", [64, 72, 1024, 1032, 2056, 4096, 4104])
@pytest.mark.parametrize("mixer", ["gla", "win"])
def test_one_row_normed_on_its_way_in(mixer, width, monkeypatch):
    mix = {"gla": gla(3, 16, 40), "win": win(2, 1, 32, 40, 11, 3, 8)}[mixer]
    cfg = config([dict(mix, mlp={"kind": "dense", "ff": 72, "limit": 7.0})], width=width, vocab=1003)
    w = O.random_weights(cfg, seed=6)
    both_ways(lambda: residuals(cfg, w, 5, 3), monkeypatch, bound(width, 72, 3 * 40, 2 * 40))


@pytest.mark.parametrize("n", [2, 8, 9])
def test_wide_sums_share_a_launch_up_to_eight_rows(n, monkeypatch):
    """A sum of more than 8192 inputs: in one launch for 2 and 8 rows, in two for 9"""
    cfg = config([dict(win(5, 1, 24, 40, 11, 3, 8), mlp={"kind": "dense", "ff": 8200, "limit": 7.0})], width=264, vocab=101)
    w = O.random_weights(cfg, seed=5)
    both_ways(lambda: residuals(cfg, w, n, 2), monkeypatch, bound(264, 8200, 5 * 40))
