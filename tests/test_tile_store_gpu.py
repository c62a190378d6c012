"""The way out of the tile GEMMs (csrc/tile_store.cuh): boxes that a TMA store clips at the last row and column, pitched outputs whose other elements
stay as they are, residuals in place, fp32 and bf16, rows that fill a warp, a tile, or neither. Against 64-bit products of the same bf16 operands."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

ACTS = {0: lambda x: x, 1: lambda x: x * torch.sigmoid(1.702 * x), 2: F.gelu}


@pytest.mark.parametrize("plan", [64, 128, 192, 256, 2])
@pytest.mark.parametrize("M,N,K,act,f32,bias,residual", [(1, 8, 64, 0, 0, 1, 1), (1, 8, 64, 0, 1, 1, 0), (31, 72, 128, 1, 0, 1, 0), (33, 200, 72, 0, 0, 0, 1), (129, 264, 128, 2, 1, 1, 1),
                                                          (300, 520, 136, 1, 0, 1, 1), (257, 1000, 64, 0, 1, 0, 0), (1030, 776, 192, 0, 0, 1, 1), (2700, 2056, 64, 1, 0, 1, 0)])
def test_rows_and_columns_at_the_edges(M, N, K, act, f32, bias, residual, plan):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    g = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rnd(*s):
        return torch.randn(*s, device="cuda", generator=g).bfloat16()

    A, W, b = rnd(M, K), (rnd(N, K) / K ** 0.5).bfloat16(), rnd(N) if bias else None
    out = torch.full((M + 2, N + 24), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    ref = A.double() @ W.double().T + (b.double() if bias else 0.0)
    ref = ACTS[act](ref)
    r, ld_r = None, 0
    if residual and f32:
        r, ld_r = rnd(M, N), N
        ref = ref + r.double()
    elif residual:   # in place
        out[:M, :N] = rnd(M, N)
        r, ld_r = out, N + 24
        ref = ref + out[:M, :N].double()
    _b2.check(lib.b2_op_gemm(P(A), K, P(W), K, P(b), P(r), ld_r, P(out), N + 24, f32, M, N, K, act, plan, _b2.stream_ptr()))
    # fp32 sums of K products, cut off every 16 of them: at most K / 16 times 2^-23 of a partial sum of size <= ~4; one bf16 rounding (2^-9); the
    # activations use the fast exponential and division (a few 2^-21 of values up to ~8)
    tol = K / 16 * 2 ** -23 * 4 + (2 ** -20 if f32 else 2 ** -8) * ref.abs().clamp(min=2 ** -6) + (2 ** -16 if act else 0.0)
    err = (out[:M, :N].double() - ref).abs()
    assert bool((err <= tol).all()), float((err - tol).max())
    assert bool((out[M:] == 7.0).all()) and bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("plan", [64, 128, 192, 256, 2])
@pytest.mark.parametrize("M", [1, 8, 31, 33, 48, 49])
@pytest.mark.parametrize("N,act,bias,residual", [(8, 0, 0, 0), (264, 1, 1, 0), (1000, 0, 0, 1)])
def test_fp32_outputs_of_a_few_rows(M, N, act, bias, residual, plan):
    test_rows_and_columns_at_the_edges(M, N, 136, act, 1, bias, residual, plan)
