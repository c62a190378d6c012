"""bf16 LayerNorm (csrc/norms.cu) in all of its register forms, at row counts around whole blocks of four and above one wave of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [256, 1024, 1280, 1536, 1792, 2048])
@pytest.mark.parametrize("rows", [1, 3, 4, 5, 577, 9232, 9233])
def test_layernorm_rows(rows, cols):
    from llava import _b2

    lib, P = _b2.init(0), _b2.ptr
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = (torch.randn(rows, cols, device="cuda", generator=g) + torch.randn(rows, 1, device="cuda", generator=g)).bfloat16()
    w, b = ((torch.randn(cols, device="cuda", generator=g) * 0.1 + c).bfloat16() for c in (1.0, 0.0))
    y = torch.full((rows + 1, cols), 7.0, device="cuda", dtype=torch.bfloat16)
    _b2.check(lib.b2_op_layernorm(P(x), P(w), P(b), P(y), rows, cols, 1e-5, _b2.stream_ptr()))
    ref = torch.nn.functional.layer_norm(x.double(), (cols,), w.double(), b.double(), 1e-5)
    # the output's rounding (8 significant bits) and fp32 statistics of up to 2048 terms of size ~2
    assert bool(((y[:rows].double() - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -16).all())
    assert bool((y[rows] == 7).all())
