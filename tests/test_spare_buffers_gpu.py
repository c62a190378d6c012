"""Scratch that only the faster paths use (csrc/seq_engine.cu, alloc_spare) on a device that is almost full: it never takes the room of what a
cache or a model cannot do without, and an engine that got none of it gives the same results on the other paths."""
import contextlib

import numpy as np
import pytest
import torch

import test_katadra_gpu as K
import test_sofopel_gpu as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def device_with(free):
    """Everything but `free` bytes of the device's memory taken"""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def prompt(eng, kv, toks):
    return eng.append_tokens(kv, 0, toks, restart=True, residuals=True)[1][0].clone()


def test_a_cache_fits_where_its_own_memory_does():
    heads, kv_heads, dim, vdim, seq = 128, 8, 64, 256, 4500
    cfg = S.config([dict(S.win(heads, kv_heads, dim, vdim, None, None, 0), mlp=None)], width=64)
    model, _ = S.build(cfg, torch.float32, max_batch=1, max_seq=64, max_rows=64)
    eng, toks = model._ensure_engine(), S.tokens_for(cfg, 50)
    first = eng.new_kv(1, 64)
    ref = prompt(eng, first, toks)
    own = kv_heads * seq * (dim + vdim) * 4 + 8 * heads * 64 * (vdim + 2) * 4   # keys and values, partial sums of a step's key splits
    spare = 6 * kv_heads * (dim + vdim) * seq                                   # bf16 parts of its keys and values: as large as the partial sums
    assert spare > 60 * MB
    again = eng.new_kv(1, 64)
    assert torch.equal(prompt(eng, again, toks), ref)   # every kernel of the lines below is loaded by now
    again.close()
    with device_with(own + 50 * MB):
        kv = eng.new_kv(1, seq)
        got = prompt(eng, kv, toks)
        torch.cuda.synchronize()
        kv.close()
    assert torch.equal(got, ref)
    first.close()
    model.invalidate_engine()


@pytest.mark.parametrize("name", ["katadra", "sofopel"])
def test_engines_without_spare_scratch(name):
    """True fp32: products, attention and recurrences of 260 tokens, all of which have a path with scratch and one without"""
    mod, cfg = (K, K.CFG_MAIN) if name == "katadra" else (S, S.CFG_MAIN)
    n = 260
    toks = mod.tokens_for(cfg, n)

    def run():
        model, w = mod.build(cfg, torch.float32, max_batch=1, max_seq=n + 4, max_rows=n)
        eng = model._ensure_engine()
        kv = eng.new_kv(1, n + 4)
        logits = eng.append_tokens(kv, 0, toks, list(range(n)), restart=True).clone()
        step = eng.decode_step(kv, torch.tensor([toks[0]], dtype=torch.int32)).clone()
        torch.cuda.synchronize()
        kv.close()
        model.invalidate_engine()
        return torch.cat([logits, step.reshape(1, -1)]), w

    with_scratch, w = run()
    with device_with(700 * MB):
        without, _ = run()
    ref = mod.O.forward(cfg, w, list(toks) + [toks[0]])
    ref = torch.as_tensor(np.asarray(ref if not isinstance(ref, tuple) else ref[0]))
    for got in (with_scratch, without):
        assert mod.err(got, ref) <= 2e-4     # the bound of the engines' own tests in true fp32
    assert not torch.equal(with_scratch, without)   # the two did take different paths


def test_a_refused_cache_leaves_the_calls_behind_it_alone():
    cfg = S.config([dict(S.win(8, 8, 128, 16, None, None, 0), mlp=None)], width=64)
    model, _ = S.build(cfg, torch.float32, max_batch=1, max_seq=64, max_rows=64)
    eng, toks = model._ensure_engine(), S.tokens_for(cfg, 50)
    kv = eng.new_kv(1, 64)
    ref = prompt(eng, kv, toks)
    with pytest.raises(RuntimeError, match="cudaMalloc"):
        eng.new_kv(1, 60_000_000)      # 245 GB of keys
    assert torch.equal(prompt(eng, kv, toks), ref)
    model.invalidate_engine()


def test_copies_of_weights_give_way_to_a_cache():
    """True fp32 on weights that are bf16 values: their bf16 copies are given back for a cache that finds no room beside them."""
    cfg = S.config([S.layer(S.win(8, 8, 128, 128, None, None, 0), {"kind": "dense", "ff": 16384, "limit": 1.25})], width=1024)
    model, _ = S.build(cfg, torch.float32, max_batch=1, max_seq=64, max_rows=64)
    eng, toks = model._ensure_engine(), S.tokens_for(cfg, 50)
    first = eng.new_kv(1, 64)
    ref = prompt(eng, first, toks)
    seq = 20000
    own = 8 * seq * (128 + 128) * 4
    copies = 3 * 16384 * 1024 * 2
    again = eng.new_kv(1, 64)
    assert torch.equal(prompt(eng, again, toks), ref)
    again.close()
    with device_with(own - copies // 2):
        kv = eng.new_kv(1, seq)
        got = prompt(eng, kv, toks)
        torch.cuda.synchronize()
        kv.close()
    assert S.err(got, ref) <= 2e-5      # three products of parts or six of them, fp32 sums in another order
    assert torch.equal(prompt(eng, first, toks), got)
    first.close()
    model.invalidate_engine()
