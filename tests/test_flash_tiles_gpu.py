"""bf16 flash attention (csrc/attention_tc.cu) against 64-bit softmax attention at the edges of its tiles (128 queries, 64 keys) and of its
rings (2 or 3 tiles), with ragged lengths, and with scores that grow along the keys so that the running output is rescaled on every tile."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def attend(q, k, v, lens, causal, scale):
    B, S, H, D = q.shape
    out = torch.zeros_like(q, dtype=torch.float64)
    for b in range(B):
        n = S if lens is None else int(lens[b])
        s = torch.einsum("shd,thd->hst", q[b].double(), k[b, :n].double()) * scale
        if causal:
            s = s.masked_fill(torch.arange(n, device=s.device) > torch.arange(S, device=s.device)[:, None], float("-inf"))
        out[b] = torch.einsum("hst,thd->shd", torch.softmax(s, -1), v[b, :n].double())
    return out


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("S", [1, 63, 64, 65, 127, 128, 129, 192, 193, 257, 577])
@pytest.mark.parametrize("growing", [False, True])
def test_tile_edges(S, D, causal, growing):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    B, H = 2, 3
    g = torch.Generator(device="cuda").manual_seed(S + D)
    q, k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    if growing:   # a common direction in q and k whose size grows along the keys: scores rise by far more than 2^8 from tile to tile
        q[..., 0] = 8.0
        k[..., 0] = torch.arange(S, device="cuda").div(16, rounding_mode="floor").clamp(max=200).bfloat16()[None, :, None]
    scale = 1 / math.sqrt(D)
    for lens in (None, torch.tensor([S, max(1, S // 2)], dtype=torch.int32, device="cuda")):
        o = torch.empty_like(q)
        _b2.check(lib.b2_op_flash_attn(P(q), P(k), P(v), P(o), P(lens), B, S, H, D, causal, scale, _b2.stream_ptr()))
        ref = attend(q, k, v, lens, causal, scale)
        # P is rounded to bf16 (2^-9 each, of weights that sum to 1) and so is the output: 2^-8 of the largest value, with room for scores of up to
        # ~150 in fp32 (2^-24 of them in the exponent)
        tol = 2 ** -8 * float(v.abs().max()) + 2 ** -8
        for b in range(B):   # rows past a causal request's length are padding
            n = S if lens is None or not causal else int(lens[b])
            assert float((o[b, :n].double() - ref[b, :n]).abs().max()) <= tol


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("H", [3, 79])
@pytest.mark.parametrize("S", [64, 80, 81, 208, 337, 400, 577])
@pytest.mark.parametrize("growing", [False, True])
def test_two_groups_and_one(S, H, D, causal, growing):
    """Few and many CTAs (tiles in turn by two groups of warps, or one), last tiles of at most 16 keys and of one more, a last query tile with warps that have no row."""
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    B = 2
    g = torch.Generator(device="cuda").manual_seed(S + D + H)
    q, k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    if growing:
        q[..., 0] = 8.0
        k[..., 0] = torch.arange(S, device="cuda").div(16, rounding_mode="floor").clamp(max=200).bfloat16()[None, :, None]
    scale = 1 / math.sqrt(D)
    for lens in (None, torch.tensor([S, max(1, S - 63)], dtype=torch.int32, device="cuda")):
        o = torch.empty_like(q)
        _b2.check(lib.b2_op_flash_attn(P(q), P(k), P(v), P(o), P(lens), B, S, H, D, causal, scale, _b2.stream_ptr()))
        ref = attend(q, k, v, lens, causal, scale)
        tol = 2 ** -8 * float(v.abs().max()) + 2 ** -8   # as above
        for b in range(B):
            n = S if lens is None or not causal else int(lens[b])
            assert float((o[b, :n].double() - ref[b, :n]).abs().max()) <= tol


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [0, 1])
def test_requests_without_keys(D, causal):
    """A length of 0 (or below) leaves its rows zeros and the other requests of the call as they are."""
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    B, S, H = 5, 130, 2
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    lens = torch.tensor([70, 0, 130, -3, 1], dtype=torch.int32, device="cuda")
    o = torch.full_like(q, 7.0)
    _b2.check(lib.b2_op_flash_attn(P(q), P(k), P(v), P(o), P(lens), B, S, H, D, causal, 1 / math.sqrt(D), _b2.stream_ptr()))
    for b, n in enumerate(lens.tolist()):
        if n <= 0:
            assert bool((o[b] == 0).all())
        else:
            ref = attend(q[b:b + 1], k[b:b + 1], v[b:b + 1], lens[b:b + 1], causal, 1 / math.sqrt(D))[0]
            rows = n if causal else S
            assert float((o[b, :rows].double() - ref[:rows]).abs().max()) <= 2 ** -8 * float(v[b].abs().max()) + 2 ** -8


@pytest.mark.parametrize("D,causal,S,B,H", [(128, 1, 704, 8, 32), (128, 0, 321, 8, 32), (64, 0, 577, 16, 16), (64, 1, 704, 8, 32), (128, 1, 128, 64, 32)])
def test_full_grids(D, causal, S, B, H):
    """Several waves of blocks, two on each multiprocessor: products are slow enough here for the softmax of the last tile to end before the product
    of the tile before it, and the output may only be read after the last one."""
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(B, S, H, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    scale = 1 / math.sqrt(D)
    for _ in range(3):
        o = torch.empty_like(q)
        _b2.check(lib.b2_op_flash_attn(P(q), P(k), P(v), P(o), None, B, S, H, D, causal, scale, _b2.stream_ptr()))
        for b in range(B):
            ref = attend(q[b:b + 1], k[b:b + 1], v[b:b + 1], None, causal, scale)
            assert float((o[b:b + 1].double() - ref).abs().max()) <= 2 ** -8 * float(v[b].abs().max()) + 2 ** -8
