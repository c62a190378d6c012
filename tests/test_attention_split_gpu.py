"""Prompt attention on the tensor cores (csrc/attention_split.cu) against the plain oracle: one attention layer in true fp32, at the edges of its
key tiles (64, or 32 for keys above 128), query tiles (128 (row, head) pairs) and head slabs (64 entries), in one piece and in portions whose
windows, kept positions and chunks start inside the cache; and the sizes next to those that stay on the fp32 pipe."""
import numpy as np
import pytest
import torch

import test_katadra_gpu as K
from oracle import sofopel_oracle as O
from test_sofopel_gpu import build, config, diff, tokens_for, win

pytestmark = pytest.mark.gpu

MLP = {"kind": "dense", "ff": 8, "limit": 7.0}
# Projections, scores and output are sums of at most 256 fp32 terms: about 2^-24 sqrt(256 / 2) = 7e-7 of their result each (2-norm), three in a row
BOUND = 2.1e-6


def check(mixer, portions, seed=0):
    cfg = config([dict(mixer, mlp=MLP)], width=64, vocab=90, mult=1.0)
    n = sum(portions)
    model, w = build(cfg, torch.float32, seed=seed, max_batch=2, max_seq=n + 3, max_rows=max(portions))
    toks = tokens_for(cfg, n, seed + 1)
    eng = model._ensure_engine()
    kv, got, at = eng.new_kv(2, n + 3), [], 0
    for p in portions:
        got.append(eng.append_tokens(kv, 1, toks[at:at + p], restart=at == 0, residuals=True)[1][0])
        at += p
    got = torch.cat(got).double().cpu().numpy()
    ref = O.forward(cfg, w, toks, return_layers=True)[1][0]
    add = ref - np.asarray(w["embed"], np.float64)[toks] * cfg["embedding"]["scale"]   # what the layer adds
    model.invalidate_engine()
    err = np.linalg.norm(got - ref) / np.linalg.norm(add)
    assert err <= BOUND, (mixer, portions, err)


@pytest.mark.parametrize("n", [15, 16, 31, 33, 63, 64, 65, 128, 129])
def test_edges_of_key_and_query_tiles(n):
    check(win(4, 1, 128, 128, None, None, 64), [n])


@pytest.mark.parametrize("n", [40, 63, 64, 65, 96, 97])
@pytest.mark.parametrize("vdim", [64, 128])
def test_edges_of_the_key_tiles_of_wide_keys(n, vdim):
    check(win(3, 1, 192, vdim, None, None, 64), [n])


# as BOUND, with the soft-cap, the query's temperature and the layer norm behind the three sums
BOUND_EXTRA = 5e-6


@pytest.mark.parametrize("dim,vdim", [(40, 64), (64, 128), (128, 64), (128, 128), (192, 64), (192, 128)])
@pytest.mark.parametrize("extra", ["cap", "bias", "both"])
@pytest.mark.parametrize("portions", [[40], [63], [64], [65], [129], [45, 20, 64]])
def test_soft_cap_and_distance_bias(dim, vdim, extra, portions):
    left = {"heads": 4, "kv_heads": 2, "dim": dim, "vdim": vdim, "bias_max": 50, "scale": dim ** -0.5, "softcap": 1e4 if extra == "bias" else 1.5,
            "q_temp": {"coef": 0.3, "every": 16}, "rel_rows": 12}
    cfg = K.config([{"type": "parallel", "mlp": None, "mixer": {"left": left, "right": {"heads": 1, "dim": 8, "decay_rank": 2}, "left_scale": 1.0, "right_scale": 0.0}}],
                   width=64, vocab=90)
    w = K.O.random_weights(cfg, seed=2)
    rel = next(k for k in w if k.endswith("left.rel"))
    w[rel] = w[rel] * 0 if extra == "cap" else (w[rel] / w[rel].std()).bfloat16().to(w[rel].dtype)
    n = sum(portions)
    model, _ = K.build(cfg, torch.float32, weights=w, max_batch=2, max_seq=n + 3, max_rows=max(portions))
    toks = K.tokens_for(cfg, n)
    eng = model._ensure_engine()
    kv, got, at = eng.new_kv(2, n + 3), [], 0
    for p in portions:
        got.append(eng.append_tokens(kv, 1, toks[at:at + p], restart=at == 0, residuals=True)[1][0])
        at += p
    got = torch.cat(got).double().cpu()
    model.invalidate_engine()
    ref = K.O.forward(cfg, w, toks, return_layers=True)[1][0].double()
    add = ref - w["embed"].double()[torch.tensor(toks)]
    assert float((got - ref).norm() / add.norm()) <= BOUND_EXTRA


@pytest.mark.parametrize("heads,kv,dim,vdim", [(1, 1, 64, 64), (2, 2, 65, 65), (3, 1, 192, 128), (5, 5, 8, 4), (6, 2, 129, 61), (7, 1, 30, 127), (2, 1, 193, 128), (2, 1, 128, 129)])
def test_head_sizes_and_groups(heads, kv, dim, vdim):
    check(win(heads, kv, dim, vdim, 40, 3, dim // 4 * 2), [70])


@pytest.mark.parametrize("size,keep", [(1, 1), (7, 0), (64, 5), (30, 100), (50, 64)])
@pytest.mark.parametrize("portions", [[150], [40, 17, 70, 16, 7], [100, 33]])
def test_windows_and_kept_positions(size, keep, portions):
    check(win(4, 2, 24, 40, size, keep, 8), portions)


@pytest.mark.parametrize("chunk", [1, 16, 64, 100])
@pytest.mark.parametrize("portions", [[150], [20, 60, 16, 41]])
def test_two_maps_in_chunks(chunk, portions):
    check(diff(4, 2, 64, 72, 3, chunk, 32), portions)


# Without soft-cap and bias, calls that see more than 256 keys run with two softmax threads a pair, the others with four
SIZES = [(64, 64), (64, 128), (128, 64), (128, 128), (192, 64), (192, 128)]


@pytest.mark.parametrize("dim,vdim", SIZES)
@pytest.mark.parametrize("portions", [[255], [256], [257], [330], [200, 65, 64]])
def test_around_the_line_between_two_and_four_softmax_threads(dim, vdim, portions):
    check(win(4, 2, dim, vdim, None, None, dim // 2), portions)


@pytest.mark.parametrize("dim,vdim", SIZES)
@pytest.mark.parametrize("size,keep", [(300, 5), (70, 64), (260, 0)])
def test_windows_over_many_keys(dim, vdim, size, keep):
    check(win(3, 1, dim, vdim, size, keep, 8), [400])


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128), (192, 128)])
@pytest.mark.parametrize("chunk", [50, 280])
@pytest.mark.parametrize("portions", [[400], [290, 110]])
def test_two_maps_in_chunks_over_many_keys(dim, vdim, chunk, portions):
    check(diff(2, 1, dim, vdim, 3, chunk, 32), portions)
