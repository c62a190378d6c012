"""True-fp32 Linears of prompt portions on the tensor cores (csrc/linear_split.cu) against the oracle: one layer and the head, at the edges of the
128-row tiles, of the 64-wide blocks of K and of tiles of 64 and 128 columns, at sizes that are no multiple of 8, and a head whose parts exceed
the scratch and go in blocks of rows."""
import numpy as np
import pytest
import torch

from oracle import sofopel_oracle as O
from test_sofopel_gpu import build, config, tokens_for, win

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def prompt(eng, toks):
    n = len(toks)
    logits, stream = eng.append_tokens(eng.new_kv(1, n + 2), 0, toks, list(range(n)), restart=True, residuals=True)
    return logits.double().cpu().numpy(), stream[0].double().cpu().numpy()


def check(width, ff, vocab, n, seed=0):
    cfg = config([dict(win(3, 1, 20, 28, None, None, 8), mlp={"kind": "dense", "ff": ff, "limit": 7.0})], width=width, vocab=vocab, mult=1.0)
    model, w = build(cfg, torch.float32, seed=seed, max_batch=1, max_seq=n + 2, max_rows=n)
    toks = tokens_for(cfg, n)
    logits, stream = prompt(model._ensure_engine(), toks)
    model.invalidate_engine()
    holds(cfg, w, toks, logits, stream, width, ff)


def holds(cfg, w, toks, logits, stream, width, ff):
    ref, layers = O.forward(cfg, w, toks, return_layers=True)
    # each product is a sum of K fp32 terms, about 2^-24 sqrt(K / 2) of a result; four follow one another (projection, scores, output / unit, head)
    k = max(width, ff, 84)
    bound = 4 * 2 ** -24 * (k / 2) ** 0.5 + 2 ** -22
    assert rel(stream, layers[0]) <= bound
    assert rel(logits, ref) <= bound


@pytest.mark.parametrize("n", [8, 9, 24, 127, 128, 129, 260])
def test_rows(n):
    check(136, 200, 150, n)


@pytest.mark.parametrize("width,ff,vocab", [(64, 64, 64), (63, 65, 129), (8, 1, 7), (200, 1000, 300), (130, 72, 8200)])
def test_sizes(width, ff, vocab):
    check(width, ff, vocab, 40)


def test_weights_in_blocks_of_rows():
    check(320, 40, 40000, 30)


# Matrices of bf16 values are multiplied as they are; one value with more bits, in the last row too, and all three parts of the matrix are
@pytest.mark.parametrize("odd", ["all", "one", "none"])
@pytest.mark.parametrize("width,ff,n", [(64, 72, 9), (136, 200, 130), (264, 1032, 300), (1032, 136, 64)])
def test_weights_with_more_bits(odd, width, ff, n):
    from llava.model import SofopelConfig, SofopelForCausalLM

    cfg = config([dict(win(3, 1, 20, 28, None, None, 8), mlp={"kind": "dense", "ff": ff, "limit": 7.0})], width=width, vocab=150, mult=1.0)
    w = {k: np.array(v, np.float32) for k, v in O.random_weights(cfg, seed=7).items()}
    for k, v in w.items():
        if odd == "all":
            v *= np.float32(1.0 + 2.0 ** -13)
        elif odd == "one":
            v[..., -1:] *= np.float32(1.0 + 2.0 ** -23)
    model = SofopelForCausalLM(SofopelConfig(**cfg), {k: torch.from_numpy(v) for k, v in w.items()}, dtype=torch.float32, max_batch=1, max_seq=n + 2, max_rows=n)
    toks = tokens_for(cfg, n)
    eng = model._ensure_engine()
    holds(cfg, w, toks, *prompt(eng, toks), width, ff)
    # a matrix that is set in a finalized model is the one that the next call multiplies with
    w["l0.mlp.down"], w["head"] = w["l0.mlp.down"][::-1].copy(), w["head"] * np.float32(0.75)
    for k in ("l0.mlp.down", "head"):
        eng.set_weight(k, torch.from_numpy(w[k]))
    holds(cfg, w, toks, *prompt(eng, toks), width, ff)
    model.invalidate_engine()


# K over clusters of 2 to 8 CTAs with a ragged last share, tiles of 256 columns
@pytest.mark.parametrize("width,ff,vocab,n", [(64, 4100, 70, 300), (136, 2056, 130, 40), (1024, 1536, 150, 600), (520, 264, 3000, 260), (2056, 72, 65, 129)])
def test_shared_out_sums_and_wide_tiles(width, ff, vocab, n):
    check(width, ff, vocab, n, seed=2)
