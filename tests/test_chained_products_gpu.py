"""Products whose second operand is what the call in front on the same stream writes (keys of a score matrix that were projected just now): the tile
GEMMs on every plan, the gated unit, and the stream-K GEMM. The first call takes few SMs for long, so that the second one's CTAs are
there early; its result has to be that of the same two calls with a synchronisation between them, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

N, K = 512, 1024     # of the second product: its W is the [N, K] output of the first


def operands(seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd(*s):
        return torch.randn(*s, device="cuda", generator=g).bfloat16()

    return rnd


def both_ways(second, seed):
    """W = X P^T into a buffer that holds something else, then second(W)"""
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    rnd = operands(seed)
    X, Pj, W = rnd(N, 8192), rnd(K, 8192) / 64, torch.empty(N, K, device="cuda", dtype=torch.bfloat16)
    outs = []
    for wait in (True, False, False, False):
        W.fill_(3.0)
        torch.cuda.synchronize()
        _b2.check(lib.b2_op_gemm(P(X), 8192, P(Pj), 8192, None, None, 0, P(W), K, 0, N, K, 8192, 0, 256, _b2.stream_ptr()))
        if wait:
            torch.cuda.synchronize()
        outs.append(second(lib, P, W, rnd))
        torch.cuda.synchronize()
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
    return outs[0]


@pytest.mark.parametrize("plan", [0, 64, 128, 192, 256, 2, 2064, 2128, 4064])
@pytest.mark.parametrize("M", [64, 600])
def test_tile_gemms(plan, M):
    from llava import _b2

    A = operands(1)(M, K)

    def second(lib, P, W, rnd):
        out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
        _b2.check(lib.b2_op_gemm(P(A), K, P(W), K, None, None, 0, P(out), N, 0, M, N, K, 0, plan, _b2.stream_ptr()))
        return out

    both_ways(second, 2)


@pytest.mark.parametrize("plan", [128, 256, 2])
def test_gated_unit(plan):
    from llava import _b2

    A = operands(1)(600, K)

    def second(lib, P, W, rnd):
        out = torch.zeros(600, N // 2, device="cuda", dtype=torch.bfloat16)
        _b2.check(lib.b2_op_gemm_glu(P(A), K, P(W), K, P(out), N // 2, 600, N // 2, K, 1.0, 0.0, 0.0, 0, None, 1, plan, _b2.stream_ptr()))
        return out

    both_ways(second, 3)


@pytest.mark.parametrize("B", [9, 40, 128])
@pytest.mark.parametrize("fp8", [False, True])
def test_stream_k(B, fp8):
    from llava import _b2

    lib = _b2.init(0)
    work = torch.zeros(lib.b2_op_gemm_skinny_workspace_bytes(B, N, 2 * K), device="cuda", dtype=torch.uint8)
    count = torch.zeros(lib.b2_op_gemm_skinny_counter_bytes(N), device="cuda", dtype=torch.uint8)
    x, ones = operands(1)(B, K), torch.ones(max(B, N), device="cuda")
    x8 = x.float().to(torch.float8_e4m3fn)

    def second(lib, P, W, rnd):
        out = torch.zeros(B, N, device="cuda", dtype=torch.float32)
        if fp8:     # the bytes of W as e4m3: [N, K] of its rows of 2 K bytes (NaN encodings among them)
            _b2.check(lib.b2_op_gemm_skinny_fp8(P(x8), K, P(ones), P(W), 2 * K, P(ones), None, 0, P(out), N, 1, B, N, K, 0, P(work), work.numel(), P(count), _b2.stream_ptr()))
            return torch.nan_to_num(out)
        _b2.check(lib.b2_op_gemm_skinny(P(x), K, P(W), K, None, 0, P(out), N, 1, B, N, K, 0, P(work), work.numel(), P(count), _b2.stream_ptr()))
        return out

    both_ways(second, 4)
