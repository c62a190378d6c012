"""Linears of 1..16 rows on streamed bf16 weights (csrc/linear_stream.cu) against the FMA kernels on the same bf16 operands: one layer of a
model, at row counts around the two column tiles of 8, input sizes around the units of 128 that the warps share, and output sizes that are no
multiple of a tile of 16."""
import pytest
import torch

from oracle import sofopel_oracle as O
from test_sofopel_gpu import config, tokens_for, win

pytestmark = pytest.mark.gpu


def bound(*sizes):
    """Both sides multiply the same bf16 operands and add up in fp32, in other orders (1e-7 of a result). That leaves the operands of the NEXT
    product equal but for the odd entry that falls on the other side of a bf16 rounding: it moves by 2^-8 of itself, and a sum over K entries
    by 2^-8 |entry| / (rms sqrt(K)). Room for one such entry of three times the rms in the smallest of the layer's sums."""
    return 3 * 2 ** -8 / min(sizes) ** 0.5


def residuals(cfg, w, n, steps):
    from llava.model import SofopelConfig, SofopelForCausalLM

    model = SofopelForCausalLM(SofopelConfig(**cfg), {k: torch.from_numpy(v).bfloat16() for k, v in w.items()}, dtype=torch.bfloat16, max_batch=2, max_seq=64,
                               max_rows=32)
    eng = model._ensure_engine()
    kv, toks = eng.new_kv(2, 64), tokens_for(cfg, n + steps)
    out = [eng.append_tokens(kv, 0, toks[:n], list(range(n)), restart=True, residuals=True)]
    out = [out[0][1].flatten().double(), out[0][0].flatten().double()]
    out += [eng.decode_step(kv, torch.tensor([t], dtype=torch.int32)).flatten().double() for t in toks[n:]]
    torch.cuda.synchronize()
    model.invalidate_engine()
    return out


@pytest.mark.parametrize("width,ff", [(64, 24), (64, 100), (72, 136), (136, 40), (264, 1032), (1160, 272)])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17])
def test_streamed_weights_equal_the_fma_kernels(width, ff, n, monkeypatch):
    cfg = config([dict(win(5, 1, 24, 40, None, None, 8), mlp={"kind": "dense", "ff": ff, "limit": 7.0})], width=width, vocab=101)
    w = O.random_weights(cfg, seed=3)
    monkeypatch.setenv("B2_SEQ_TC", "1")
    got = residuals(cfg, w, n, 2)
    monkeypatch.setenv("B2_SEQ_TC", "0")
    ref = residuals(cfg, w, n, 2)
    for a, b in zip(got, ref):
        assert float((a - b).norm() / b.norm()) <= bound(width, ff, 5 * 40)
