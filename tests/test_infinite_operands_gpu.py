"""Operands that three bf16 parts do not hold (infinities, finite values that round to infinity in bf16) in the fp32 kernels that cut their operands
into parts (csrc/linear_split.cu, csrc/attention_split.cu): results are those of fp32 products, and nothing leaks into rows and columns that do
not meet such an operand."""
import numpy as np
import pytest
import torch

from oracle import sofopel_oracle as O
from test_sofopel_gpu import config, diff, tokens_for, win

pytestmark = pytest.mark.gpu

HUGE = 2.0 ** 127 * 1.75     # representable in bf16; twice it is not a finite fp32
BOUND = 4e-6                 # as the kernels' own tests: a few sums of up to 256 fp32 terms


def run(cfg, w, toks, dtype=torch.float32, portions=None):
    from llava.model import SofopelConfig, SofopelForCausalLM

    n = len(toks)
    model = SofopelForCausalLM(SofopelConfig(**cfg), {k: torch.from_numpy(np.asarray(v, np.float32)) for k, v in w.items()}, dtype=dtype, max_batch=1,
                               max_seq=n + 2, max_rows=n)
    eng = model._ensure_engine()
    kv, logits, stream, at = eng.new_kv(1, n + 2), [], [], 0
    for p in portions or [n]:
        lg, rs = eng.append_tokens(kv, 0, toks[at:at + p], list(range(p)), restart=at == 0, residuals=True)
        logits.append(lg)
        stream.append(rs[0])
        at += p
    out = torch.cat(logits).double().cpu().numpy(), torch.cat(stream).double().cpu().numpy()
    model.invalidate_engine()
    return out


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", [9, 130])
@pytest.mark.parametrize("vocab", [90, 8200])
def test_weights_that_have_no_parts(n, vocab):
    cfg = config([dict(win(2, 1, 16, 16, None, None, 0), mlp=None)], width=72, vocab=vocab, mult=1.0)
    w = O.random_weights(cfg, seed=1)
    head = w["head"].copy()
    head[5, 3], head[vocab - 1, 71] = np.inf, -np.inf
    head[7, 9] = np.float32(3.4e38)        # finite in fp32, infinite in bf16
    head[8, :] = 0
    head[8, 2], head[8, 4] = np.float32(3.399e38), np.float32(-3.399e38)
    w["head"] = head
    toks = tokens_for(cfg, n)
    got, stream = run(cfg, w, toks)
    clean = dict(w, head=np.where(np.isfinite(head) & (np.abs(head) < 1e38), head, 0))
    ref, layers = O.forward(cfg, clean, toks, return_layers=True)
    x = ref_norm(cfg, w, layers[0])
    assert np.array_equal(got[:, 5], np.where(x[:, 3] > 0, np.inf, -np.inf))
    assert np.array_equal(got[:, vocab - 1], np.where(x[:, 71] > 0, -np.inf, np.inf))
    big = x[:, 9] * np.float64(head[7, 9])
    assert np.array_equal(np.isinf(got[:, 7]), np.abs(big) >= 2.0 ** 128) and np.array_equal(np.sign(got[:, 7]), np.sign(big))
    fits = np.abs(big) < 2.0 ** 127
    assert fits.any() and np.abs(got[fits, 7] - big[fits]).max() <= 4e-6 * np.float64(head[7, 9])
    both = (x[:, 2] - x[:, 4]) * np.float64(head[8, 2])
    fits = (np.maximum(np.abs(x[:, 2]), np.abs(x[:, 4])) < 0.9) & (np.abs(both) < 2.0 ** 127)     # both products and their sum are finite
    assert np.isfinite(got[fits, 8]).all() and (np.abs(got[fits, 8] - both[fits]) <= 4e-6 * np.float64(head[8, 2])).all()
    others = [c for c in range(vocab) if c not in (5, 7, 8, vocab - 1)]
    assert rel(got[:, others], ref[:, others]) <= BOUND and rel(stream, layers[0]) <= BOUND


def ref_norm(cfg, w, x):
    return O.rms_norm(x, np.asarray(w["final.norm"], np.float64), float(cfg["norm"]["eps"]))


def special_token(cfg, seed):
    """Weights and a prompt in which entry 0 of the normed stream is positive for one token, at position 21, and zero for the others, and entry 1 is
    positive for all"""
    w = O.random_weights(cfg, seed=seed)
    e = w["embed"].copy()
    e[:, 0], e[3, 0], e[:, 1] = 0, 2, 1
    w["embed"] = e
    w["l0.norm1"] = np.ones_like(w["l0.norm1"])
    toks = [t if t != 3 else 4 for t in tokens_for(cfg, 90, seed + 1)]
    toks[21] = 3
    return w, toks


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("portions", [[90], [20, 70], [30, 60]])
@pytest.mark.parametrize("chunk", [None, 25])
def test_a_key_with_an_infinite_entry_and_a_score_of_minus_infinity(chunk, portions, dtype):
    """Every other token's query looks the other way, so the key is as good as absent, and the rows that see it are finite"""
    cfg = config([dict(diff(2, 1, 64, 72, None, chunk, 0), mlp=None)], width=64, vocab=90, mult=1.0)
    w, toks = special_token(cfg, 5)
    k, q = w["l0.mix.k"].copy(), w["l0.mix.q"].copy()
    k[0], q[0], q[2 * 64] = 0, 0, 0            # first entry of the first map's key, and of the first map's query of both heads
    k[0, 0], q[0, 1], q[2 * 64, 1] = HUGE, -1, -1
    w["l0.mix.k"], w["l0.mix.q"] = k, q
    _, stream = run(cfg, w, toks, dtype, portions)
    ref = O.forward(cfg, w, toks, return_layers=True)[1][0]
    assert np.isfinite(stream).all()
    assert rel(stream, ref) <= (BOUND if dtype == torch.float32 else 1e-2)


@pytest.mark.parametrize("portions", [[90], [45, 45]])
@pytest.mark.parametrize("chunk", [None, 25])
def test_rows_that_do_not_see_an_infinite_value(chunk, portions):
    cfg = config([dict(diff(2, 1, 64, 72, None, chunk, 0), mlp=None)], width=64, vocab=90, mult=1.0)
    w, toks = special_token(cfg, 6)
    v = w["l0.mix.v"].copy()
    v[1] = 0
    v[1, 0] = HUGE
    w["l0.mix.v"] = v
    _, stream = run(cfg, w, toks, portions=portions)
    ref = O.forward(cfg, w, toks, return_layers=True)[1][0]
    unseen = [i for i in range(90) if i < 21 or (chunk is not None and i // chunk != 21 // chunk)]
    assert rel(stream[unseen], ref[unseen]) <= BOUND
    seen = [i for i in range(90) if i not in unseen]
    assert not np.isfinite(stream[seen]).all(axis=1).any()     # an infinite head output has no finite root mean square
