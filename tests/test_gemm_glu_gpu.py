"""Both products of a gated feed-forward and their unit in one GEMM (csrc/gemm_tcgen05.cu, csrc/gemm_2cta.cu) against 64-bit products of the same
bf16 operands: widths that end inside a tile's 64 gate rows, ragged rows and K, every plan, each kind of unit, and rows grouped by expert."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def unit(x, ff, slope, limit, shift, kind):
    g, u = x[:, :ff], x[:, ff:]
    if limit > 0:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    a = 0.5 * g * (1 + torch.tanh(math.sqrt(2 / math.pi) * (g + 0.044715 * g ** 3))) if kind else g * torch.sigmoid(slope * g)
    return a * (u + shift)


def close(out, ref, pre, K):
    # fp32 sums of K products, cut off every 16 of them (a partial sum is at most ~4 here; the unit's slope is at most 1.1 (|u| + 1) + |a|, below 8),
    # and one rounding to bf16
    tol = K / 16 * 2 ** -23 * 4 * 8 + 2 ** -8 * ref.abs().clamp(min=2 ** -6)
    assert bool(((out - ref).abs() <= tol).all()), float(((out - ref).abs() - tol).max())


@pytest.mark.parametrize("plan", [0, 2, 128, 256])
@pytest.mark.parametrize("M,ff,K", [(17, 8, 64), (41, 136, 520), (128, 64, 2048), (129, 72, 576), (257, 264, 1000), (600, 1000, 1024), (1025, 640, 256)])
@pytest.mark.parametrize("slope,limit,shift,kind", [(1.0, 0.0, 0.0, 0), (1.702, 1.5, 1.0, 0), (1.0, 0.0, 0.0, 1)])
def test_glu(M, ff, K, slope, limit, shift, kind, plan):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    g = torch.Generator(device="cuda").manual_seed(M + ff + K)
    A = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    W = (torch.randn(2 * ff, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    out = torch.full((M + 1, ff), 7.0, device="cuda", dtype=torch.bfloat16)
    _b2.check(lib.b2_op_gemm_glu(P(A), K, P(W), K, P(out), ff, M, ff, K, slope, limit, shift, kind, None, 1, plan, _b2.stream_ptr()))
    pre = A.double() @ W.double().T
    close(out[:M].double(), unit(pre, ff, slope, limit, shift, kind), pre, K)
    assert bool((out[M] == 7.0).all())


@pytest.mark.parametrize("ff,K,plan", [(72, 512, 0), (136, 1024, 128), (264, 256, 256)])
def test_grouped(ff, K, plan):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    groups, tiles = 3, [2, 0, -1, 1, 2]
    g = torch.Generator(device="cuda").manual_seed(ff)
    M = 128 * len(tiles)
    A = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    W = (torch.randn(groups, 2 * ff, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    out = torch.full((M, ff), 7.0, device="cuda", dtype=torch.bfloat16)
    tg = torch.tensor(tiles, device="cuda", dtype=torch.int32)
    _b2.check(lib.b2_op_gemm_glu(P(A), K, P(W), K, P(out), ff, M, ff, K, 1.0, 0.0, 0.0, 0, P(tg), groups, plan, _b2.stream_ptr()))
    for i, e in enumerate(tiles):
        rows = slice(128 * i, 128 * i + 128)
        if e < 0:
            assert bool((out[rows] == 7.0).all())
        else:
            pre = A[rows].double() @ W[e].double().T
            close(out[rows].double(), unit(pre, ff, 1.0, 0.0, 0.0, 0), pre, K)


def test_other_entry_refuses_the_unit():
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    x = torch.zeros(128, 128, device="cuda", dtype=torch.bfloat16)
    assert lib.b2_op_gemm(P(x), 128, P(x), 128, None, None, 0, P(x), 128, 0, 128, 128, 128, 5, 0, _b2.stream_ptr()) != 0
