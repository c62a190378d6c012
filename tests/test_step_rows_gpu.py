"""The small kernels around a decode step at the widths where their 16-byte paths begin and end: greedy selection (ties, NaN, -inf, odd
vocabularies), group norms of every width, and steps fed from and read into device and host memory."""
import ctypes as C

import numpy as np
import pytest
import torch

import test_sofopel_gpu as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 3, 4, 5, 31, 1024, 4095, 4096, 4097, 32000, 32768, 32771, 50257])
@pytest.mark.parametrize("fill", ["random", "ties", "nan", "neginf"])
def test_first_of_the_largest(V, fill):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    g = torch.Generator(device="cuda").manual_seed(V)
    B = 3
    x = torch.randn(B, V, device="cuda", generator=g)
    if fill == "ties":
        x = x.mul(2).round()
    elif fill == "nan":
        x[torch.rand(B, V, device="cuda", generator=g) < 0.5] = float("nan")
    elif fill == "neginf":
        x[:, : V - 1] = float("-inf")
    want = torch.where(x.isnan(), torch.full_like(x, float("-inf")), x)
    # the first of the largest; a row of -inf alone gives the first entry that is a number
    want = torch.stack([(r == r.max()).logical_and(~q.isnan()).float().argmax() for r, q in zip(want, x)])
    tok = torch.full((B,), -1, device="cuda", dtype=torch.int32)
    _b2.check(lib.b2_op_sample(P(x), B, V, C.byref(_b2.Sampling(0, 1.0, 1.0, 0, 0)), 0, P(tok), _b2.stream_ptr()))
    assert tok.tolist() == want.tolist()


@pytest.mark.parametrize("vdim", [4, 6, 124, 128, 132, 256, 260, 512, 516])
def test_group_norm_widths(vdim):
    cfg = S.config([S.layer(S.gla(3, 16, vdim), None)], width=64)
    model, w = S.build(cfg, torch.float32, max_batch=1, max_seq=16, max_rows=8)
    toks = S.tokens_for(cfg, 6)
    eng = model._ensure_engine()
    got = eng.append_tokens(eng.new_kv(1, 16), 0, toks, restart=True, residuals=True)[1][0].cpu().double()
    ref = torch.as_tensor(np.asarray(S.O.forward(cfg, w, toks, return_layers=True)[1][0])).double()
    # sums of up to heads * vdim fp32 terms, 2^-24 of a term each, with room for rows smaller than their terms
    assert float(((got - ref).norm(dim=-1) / ref.norm(dim=-1)).max()) <= 2 ** -20


@pytest.mark.parametrize("width", [40, 64, 1160])
def test_steps_from_and_into_any_memory(width):
    cfg = S.config([S.layer(S.GLA, None)], width=width, vocab=101)
    model, _ = S.build(cfg, torch.bfloat16, max_batch=3, max_seq=16, max_rows=8)
    eng = model._ensure_engine()
    kv = eng.new_kv(3, 16)
    got = []
    for odd in (False, True):
        for slot in range(3):
            eng.append_tokens(kv, slot, S.tokens_for(cfg, 4, seed=slot), restart=True)
        fed = torch.tensor([7, 8, 9, 10], dtype=torch.int32)
        fed = fed[1:] if odd else fed.cuda()[1:]   # host memory, and device memory that no 16-byte boundary begins
        out = torch.empty(3 * 101 + 1, device="cuda")[int(odd):][: 3 * 101]   # a result that begins on a 16-byte boundary, and one that does not
        nxt = torch.empty(3, dtype=torch.int32, device="cpu" if odd else "cuda")
        from llava import _b2
        P = _b2.ptr
        _b2.check(eng.lib.b2_decode_step_slots(eng.handle, kv.handle, P(fed), 3, 0, P(out), P(nxt), _b2.stream_ptr()))
        got.append((out.view(3, 101).clone(), nxt.cpu()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert torch.equal(got[0][0].argmax(-1).cpu().int(), got[0][1])


@pytest.mark.parametrize("n", [1, 7, 130])
def test_residuals_and_wanted_rows_of_any_layout(n):
    """Residual rows into a buffer that no 16-byte boundary begins and one that does; up to 128 wanted rows as kernel parameters,
    more of them as a copy."""
    from llava import _b2

    cfg = S.config([S.layer(S.GLA, None), S.layer(S.GLA, None)], width=40, vocab=101)
    model, _ = S.build(cfg, torch.bfloat16, max_batch=1, max_seq=160, max_rows=160)
    eng, P = model._ensure_engine(), _b2.ptr
    kv, toks = eng.new_kv(1, 160), S.tokens_for(cfg, n)
    ctoks = (C.c_int32 * n)(*toks)
    size = 2 * n * 40
    got = []
    for at, k in ((0, n), (1, n), (4, 1), (2, 1)):
        want = list(range(n))[-k:]
        resid, logits = torch.full((size + 8,), 7.0, device="cuda"), torch.empty(k, 101, device="cuda")
        _b2.check(eng.lib.b2_append_tokens(eng.handle, kv.handle, 0, ctoks, n, 1, (C.c_int32 * k)(*want), k, P(logits), P(resid[at:]), _b2.stream_ptr()))
        assert resid[:at].eq(7).all() and resid[at + size:].eq(7).all()
        got.append((resid[at:at + size].clone(), logits[-1:].clone(), logits))
    assert all(torch.equal(g[0], got[0][0]) for g in got)
    assert torch.equal(got[0][2], got[1][2]) and torch.equal(got[2][1], got[3][1])
    # (one row of logits is a product of its own: bf16 operands, fp32 sums in another order)
    assert torch.allclose(got[0][1], got[2][1], atol=2 ** -8 * float(got[0][1].abs().max()))


@pytest.mark.parametrize("width", [500, 512, 516, 1022, 1024, 1028, 2048, 2052])
def test_rows_normed_in_registers(width):
    """LayerNorm onto the residual stream and in front of the head, at the widths where its register forms begin and end."""
    import test_katadra_gpu as K

    cfg = K.config([K.MAMBA], width=width)
    model, w = K.build(cfg, torch.float32, max_batch=1)
    toks = K.tokens_for(cfg, 11)
    logits, hidden = model.forward(torch.tensor([toks]), output_hidden_states=True)
    ref, layers = K.O.forward(cfg, w, toks, return_layers=True)
    # fp32 sums of up to 2052 terms (2^-24 of a term each, growing with the root of their number) in two products and the norms behind them
    assert K.err(hidden[0, 0], layers[0]) <= 2 ** -24 * 4 * 2052 ** 0.5
    assert K.err(logits[0], ref) <= 2 ** -24 * 8 * 2052 ** 0.5


@pytest.mark.parametrize("name", ["gla", "diff", "win", "memory"])
def test_one_row_steps_where_every_row_counts_as_a_tensor_core_one(name, monkeypatch):
    """B2_SEQ_TC_MIN_ROWS=1: the step of one row streams its fp32 rows all the same, so nothing in front of it may leave bf16 rows alone."""
    import test_ramosun_gpu as R

    if name == "memory":
        mod, cfg = R, R.CFG_MAIN
    else:
        mix = {"gla": S.gla(2, 32, 32), "diff": S.diff(2, 1, 32, 32, None, None, 32), "win": S.win(2, 1, 32, 32, None, None, 32)}[name]
        mod, cfg = S, S.config([S.layer(mix, {"kind": "dense", "ff": 64, "limit": 1.25})] * 2, width=64)
    toks, got = mod.tokens_for(cfg, 9), []
    for rows in ("1", "2"):
        monkeypatch.setenv("B2_SEQ_TC_MIN_ROWS", rows)
        model, _ = mod.build(cfg, torch.bfloat16, max_batch=1, max_seq=32, max_rows=16)
        eng = model._ensure_engine()
        kv = eng.new_kv(1, 32)
        eng.append_tokens(kv, 0, toks[:5], restart=True)
        got.append(torch.cat([eng.decode_step(kv, torch.tensor([t], dtype=torch.int32)).clone().view(1, -1) for t in toks[5:]]))
        model.invalidate_engine()
    assert torch.equal(got[0], got[1])
