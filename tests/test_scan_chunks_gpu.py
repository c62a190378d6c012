"""Recurrences of long prompts, walked in chunks side by side (csrc/recurrent.cu): every form of the recurrence, whole prompts around the lengths
at which chunks begin (192 tokens), end unevenly and reach their largest number, against the same prompt in portions that are walked in one
piece, with a slot that already holds a state, and against the oracles."""
import numpy as np
import pytest
import torch

import test_katadra_gpu as K
import test_pefivik_gpu as P
import test_sofopel_gpu as S

pytestmark = pytest.mark.gpu

MAMBA = {"type": "mamba2", "mlp": None, "mixer": {"heads": 6, "vdim": 70, "state": 130, "groups": 2, "conv": 4, "norm_groups": 3}}
RWKV = {"type": "parallel", "mlp": None,
        "mixer": {"left": {"heads": 2, "kv_heads": 1, "dim": 8, "vdim": 8, "bias_max": 12, "scale": 0.4, "softcap": 3.0, "q_temp": {"coef": 0.25, "every": 4}, "rel_rows": 6},
                  "right": {"heads": 3, "dim": 72, "decay_rank": 5}, "left_scale": 0.0, "right_scale": 1.0}}
LAYERS = {
    "mamba2": (K, K.config([K.MAMBA])), "mamba2_wide": (K, K.config([MAMBA], width=64)), "mamba2_odd": (K, K.config([K.MAMBA_ODD], width=50)),
    "rwkv": (K, K.config([RWKV], width=64)), "rwkv_odd": (K, K.config([K.PAR_ODD], width=90)),
    "hgrn2": (P, P.config([P.layer(P.HG_BIG, None)], width=64)), "hgrn2_odd": (P, P.config([P.layer(P.HG_ODD, None)], width=50)),
    "gla": (S, S.config([S.layer(S.GLA, None)], width=64)), "gla_odd": (S, S.config([S.layer(S.GLA_ODD, None)], width=50)),
    "gla_wide": (S, S.config([S.layer(S.GLA_WIDE, None)], width=56)),
}


def stream(eng, kv, toks, cuts):
    out, at = [], 0
    for c in cuts:
        out.append(eng.append_tokens(kv, 1, toks[at:at + c], restart=at == 0, residuals=True)[1][0])
        at += c
    assert at == len(toks)
    return torch.cat(out).double()


def rel(a, b):
    return float(((a - b).norm(dim=-1) / b.norm(dim=-1)).max())


@pytest.mark.parametrize("name", list(LAYERS))
def test_chunks_equal_one_piece(name):
    mod, cfg = LAYERS[name]
    model, _ = mod.build(cfg, torch.float32, max_batch=2, max_seq=1100, max_rows=1100)
    eng = model._ensure_engine()
    kv = eng.new_kv(2, 1100)
    for n in (191, 192, 193, 209, 512, 1033):
        toks = mod.tokens_for(cfg, n, seed=n)
        small = [100] * (n // 100) + ([n % 100] if n % 100 else [])
        # both are the same sums of up to n fp32 terms in another order: 2^-24 sqrt(n) of a row each, with room for rows smaller than their terms
        bound = 2 ** -21 * n ** 0.5
        one = stream(eng, kv, toks, small)
        assert rel(stream(eng, kv, toks, [n]), one) <= bound, n
        assert rel(stream(eng, kv, toks, [7, n - 7]), one) <= bound, n          # the first chunk starts from a state


@pytest.mark.parametrize("name", ["mamba2", "rwkv", "hgrn2", "gla"])
def test_chunks_against_the_oracle(name):
    mod, cfg = LAYERS[name]
    n = 260
    model, w = mod.build(cfg, torch.float32, max_batch=2, max_seq=n + 4, max_rows=n)
    eng = model._ensure_engine()
    toks = mod.tokens_for(cfg, n)
    got = stream(eng, eng.new_kv(2, n + 4), toks, [n]).cpu()
    ref = mod.O.forward(cfg, w, toks) if mod is P else mod.O.forward(cfg, w, toks, return_layers=True)
    ref = torch.as_tensor(np.asarray(ref[1][0])).double()
    assert rel(got, ref) <= 2 ** -21 * n ** 0.5


# Blocks of 64 tokens on the tensor cores (csrc/scan_blocks.cu): key sizes of one and two blocks of 64 and parts of one, value sizes around tiles of 128
# columns, prompts that end inside a block, and one whose blocks exceed the scratch and goes in pieces
def rwkv(heads, dim):
    lay = {**RWKV, "mixer": {**RWKV["mixer"], "right": {"heads": heads, "dim": dim, "decay_rank": 5}}}
    return K, K.config([lay], width=64)


def hgrn2(heads, dim, vdim):
    return P, P.config([P.layer({"type": "hgrn2", "mixer": {"heads": heads, "dim": dim, "vdim": vdim}}, None)], width=64)


def gla(heads, dim, vdim):
    return S, S.config([S.layer(S.gla(heads, dim, vdim), None)], width=64)


BLOCKS = {"rwkv_64": rwkv(2, 64), "rwkv_72": rwkv(3, 72), "rwkv_128": rwkv(1, 128), "hgrn2": hgrn2(2, 128, 64), "hgrn2_part": hgrn2(3, 44, 132), "gla_small": gla(3, 16, 24),
          "gla": gla(2, 128, 256), "gla_part": gla(3, 68, 4)}


@pytest.mark.parametrize("name", list(BLOCKS))
def test_blocks_equal_small_portions(name):
    mod, cfg = BLOCKS[name]
    model, _ = mod.build(cfg, torch.float32, max_batch=2, max_seq=700, max_rows=700)
    eng = model._ensure_engine()
    kv = eng.new_kv(2, 700)
    for n in (319, 320, 448, 449, 511, 577, 640):
        toks = mod.tokens_for(cfg, n, seed=n)
        one = stream(eng, kv, toks, [100] * (n // 100) + ([n % 100] if n % 100 else []))
        bound = 2 ** -21 * n ** 0.5
        assert rel(stream(eng, kv, toks, [n]), one) <= bound, n
        assert rel(stream(eng, kv, toks, [50, n - 50]), one) <= bound, n


def test_blocks_in_pieces():
    mod, cfg = gla(64, 128, 256)   # 16 MB a block of tokens
    n = 650
    model, _ = mod.build(cfg, torch.float32, max_batch=2, max_seq=n, max_rows=n)
    eng = model._ensure_engine()
    kv = eng.new_kv(2, n)
    toks = mod.tokens_for(cfg, n)
    assert rel(stream(eng, kv, toks, [n]), stream(eng, kv, toks, [50] * 13)) <= 2 ** -21 * n ** 0.5


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.0e38])
@pytest.mark.parametrize("name", ["rwkv_64", "hgrn2", "gla"])
def test_a_row_that_is_no_number_reaches_no_earlier_one(name, value):
    mod, cfg = BLOCKS[name]
    n, at, tok = 512, 300, 3
    w = mod.O.random_weights(cfg, seed=1)
    w["embed"][tok] = value   # (an array, or a tensor)
    model, _ = mod.build(cfg, torch.float32, weights=w, max_batch=2, max_seq=n, max_rows=n)
    eng = model._ensure_engine()
    kv = eng.new_kv(2, n)
    toks = [t if t != tok else 4 for t in mod.tokens_for(cfg, n)]
    toks[at] = tok
    got, ref = stream(eng, kv, toks, [n]), stream(eng, kv, toks, [100] * 5 + [12])
    assert torch.equal(got.isnan(), ref.isnan()) and not got[:at].isnan().any()
    assert rel(got[:at], ref[:at]) <= 2 ** -21 * n ** 0.5
