"""Split attention of a decode step (decode_attn_kernel, csrc/attention.cu) against 64-bit softmax attention at the edges of its ring: stages of 24 keys,
two of them, in 1 to 16 splits, with empty splits and with scores that grow from stage to stage."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsplit", [1, 2, 3, 16])
@pytest.mark.parametrize("growing", [False, True])
def test_decode_attention_tiles(nsplit, growing):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    lens = [0, 1, 7, 8, 22, 23, 24, 25, 47, 48, 49, 71, 72, 73, 96, 383, 384, 400, 1000]
    B, H, D, Smax = len(lens), 3, 128, max(lens) + 1
    g = torch.Generator(device="cuda").manual_seed(nsplit)
    qkv, kc, vc = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((B, 3, H, D), (B, H, Smax, D), (B, H, Smax, D)))
    # with this base the rotation leaves elements 32..63 and 96..127 as they are (angles below 1e-11); q has no others
    theta = 1e30
    qkv[:, 0, :, :32], qkv[:, 0, :, 64:96] = 0, 0
    if growing:
        qkv[:, 0, :, 40] = 8.0
        kc[..., 40] = torch.arange(Smax, device="cuda").div(8, rounding_mode="floor").bfloat16()
    kc0, vc0 = kc.clone(), vc.clone()
    cur = torch.tensor(lens, device="cuda", dtype=torch.int32)
    scratch = torch.zeros(lib.b2_op_decode_attn_scratch_bytes(B, H, nsplit), device="cuda", dtype=torch.uint8)
    out = torch.empty(B, H, D, device="cuda", dtype=torch.bfloat16)
    scale = 1 / math.sqrt(D)
    for _ in range(2):   # the counters of the splits reset themselves
        out.fill_(7.0)
        _b2.check(lib.b2_op_decode_attn(P(qkv), P(kc), P(vc), P(cur), P(out), P(scratch), B, H, Smax, nsplit, theta, scale, _b2.stream_ptr()))
        for b, n in enumerate(lens):
            k = torch.cat([kc0[b, :, :n], qkv[b, 1][:, None]], 1).double()
            v = torch.cat([vc0[b, :, :n], qkv[b, 2][:, None]], 1).double()
            s = torch.einsum("hd,hnd->hn", qkv[b, 0].double(), k) * scale
            ref = torch.einsum("hn,hnd->hd", torch.softmax(s, -1), v)
            # output rounded to bf16 (8 significant bits: at most 2^-8 of it); scores of up to ~800 in fp32: 128 products summed in any order, 2^-24 of each partial sum, into the exponent
            # (a factor of up to 2^-24 * 128 * 2 relative for the common ones), weights that sum to 1 and values of up to ~5
            tol = 2 ** -8 * ref.abs() + (2 ** -24 * 64 * float(s.abs().max()) + 2 ** -18) * float(v.abs().max())
            assert bool(((out[b].double() - ref).abs() <= tol).all()), (n, float(((out[b].double() - ref).abs() - tol).max()))
            # row n is written, and nothing else
            assert torch.equal(vc[b, :, n], qkv[b, 2]) and torch.equal(kc[b, :, n, 32:64], qkv[b, 1, :, 32:64])
            assert torch.equal(kc[b, :, :n], kc0[b, :, :n]) and torch.equal(kc[b, :, n + 1:], kc0[b, :, n + 1:])


@pytest.mark.parametrize("nsplit", [7, 8, 9])
def test_splits_meet_in_groups_of_eight(nsplit):
    test_decode_attention_tiles(nsplit, True)
