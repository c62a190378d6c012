"""The GEMM whose K is cut over a cluster (csrc/gemm_splitk.cu) against 64-bit products of the same bf16 operands, at the edges of its tiles and
k-slices, with every epilogue, in every plan and through the rule that chooses one."""
import json
import re

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

ACTS = {0: lambda x: x, 1: lambda x: x * torch.sigmoid(1.702 * x), 2: F.gelu}


def product(A, W, bias, residual, f32, act, plan):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    (M, K), N = A.shape, W.shape[0]
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    _b2.check(lib.b2_op_gemm(P(A), K, P(W), K, P(bias), P(residual), N, P(out), N, int(f32), M, N, K, act, plan, _b2.stream_ptr()))
    return out.float()


@pytest.mark.parametrize("plan", [2064, 4064, 2128, 4128, 0])
@pytest.mark.parametrize("M,N,K,act,f32,bias,residual", [(1, 8, 512, 0, 1, 0, 0), (127, 136, 520, 1, 0, 1, 0), (129, 64, 576, 2, 0, 1, 1), (40, 2048, 2048, 0, 1, 1, 0),
                                                          (257, 1000, 1000, 0, 0, 1, 1), (577, 1024, 4096, 0, 0, 1, 1)])
def test_split_k(M, N, K, act, f32, bias, residual, plan):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rnd(*s):
        return torch.randn(*s, device="cuda", generator=g).bfloat16()

    A, W, b, r = rnd(M, K), (rnd(N, K) / K ** 0.5).bfloat16(), rnd(N) if bias else None, rnd(M, N) if residual else None
    ref = A.double() @ W.double().T + (b.double() if bias else 0.0)
    ref = ACTS[act](ref) + (r.double() if residual else 0.0)
    out = product(A, W, b, r, f32, act, plan).double()
    # fp32 sums of K products, cut off every 16 of them: at most K / 16 times 2^-23 of a partial sum of size <= ~4; one bf16 rounding (2^-9); the
    # activations use the fast exponential and division (a few 2^-21 of values up to ~8)
    tol = K / 16 * 2 ** -23 * 4 + (0.0 if f32 else 2 ** -8) * ref.abs().clamp(min=2 ** -6) + (2 ** -16 if act else 0.0)
    assert bool(((out - ref).abs() <= tol).all()), float(((out - ref).abs() - tol).max())


@pytest.mark.parametrize("M,N,K,act,f32,bias,residual", [(1154, 1024, 4096, 0, 0, 1, 1), (1153, 1000, 4104, 1, 0, 1, 0), (16, 5120, 2568, 0, 1, 0, 0), (500, 1160, 2568, 2, 0, 1, 1)])
def test_split_in_three(M, N, K, act, f32, bias, residual):
    """Tiles of 256 columns (the first two) and of 128 whose column groups don't divide by three, through the rule."""
    test_split_k(M, N, K, act, f32, bias, residual, 0)


@pytest.mark.parametrize("M,N,K,bn", [(1154, 1024, 4096, 256), (1153, 1000, 4104, 256), (16, 5120, 2568, 128), (500, 1160, 2568, 128)])
def test_the_rule_takes_three_slices_there(M, N, K, bn, tmp_path):
    """The shapes of the test above are those of the plans that it means: no plan number names these."""
    A, W = (torch.zeros(n, K, device="cuda", dtype=torch.bfloat16) for n in (M, N))
    product(A, W, None, None, False, 0, 0)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        product(A, W, None, None, False, 0, 0)
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    ran = [e for e in json.load(open(tmp_path / "trace.json"))["traceEvents"] if e.get("cat") == "kernel" and "gemm" in e["name"]]
    assert len(ran) == 1 and re.search(r"gemm_splitk_kernel<(\(int\))?%d\b" % bn, ran[0]["name"]), [e["name"] for e in ran]
    grid = ran[0]["args"]["grid"]
    assert grid[0] * grid[1] * grid[2] == 3 * -(-M // 128) * -(-N // bn)


def test_plans_that_do_not_fit_are_refused():
    A = torch.zeros(16, 128, device="cuda", dtype=torch.bfloat16)
    W = torch.zeros(64, 128, device="cuda", dtype=torch.bfloat16)
    for plan in (4064, 3064, 2032):     # more slices than blocks of 64, no such cluster, no such tile: turned down on the host, nothing is launched
        with pytest.raises(ValueError):
            product(A, W, None, None, True, 0, plan)
