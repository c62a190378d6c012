"""Short prompt portions through latent attention: which of its two forms a portion takes (csrc/seq_engine.cu, latent_per_head), told from the
bits of either form, forced; and both against the plain oracle. A portion below 64 rows makes per-head keys and values only where that is the faster
form: not in many small pieces, and not where the latent is narrow beside the heads' keys and values that the fp32 pipe would then read."""
import pytest
import torch

import test_pefivik_gpu as P

pytestmark = pytest.mark.gpu


def lat(heads, dim, vdim, rank):
    return {"type": "latent_attention", "mixer": {"heads": heads, "dim": dim, "vdim": vdim, "kv_rank": rank, "scale": dim ** -0.5}}


# heads, dim, vdim, rank, rows of the workspace, positions in front, rows, form
CASES = [
    (4, 16, 16, 64, 400, 300, 8, "absorbed"), (4, 16, 16, 64, 400, 300, 9, "per head"), (4, 16, 16, 64, 400, 300, 63, "per head"),
    (4, 32, 32, 24, 400, 300, 15, "absorbed"), (4, 32, 32, 24, 400, 300, 16, "per head"), (4, 32, 32, 24, 400, 300, 64, "per head"),
    (4, 16, 16, 64, 32, 300, 9, "absorbed"), (4, 16, 16, 64, 32, 300, 31, "absorbed"), (4, 16, 16, 64, 64, 300, 64, "per head"),
    (2, 200, 136, 40, 400, 300, 20, "absorbed"), (2, 200, 136, 40, 400, 0, 20, "per head"), (2, 200, 136, 40, 400, 300, 70, "per head"),
    (2, 200, 136, 344, 400, 300, 12, "absorbed"), (1, 16, 16, 64, 400, 300, 15, "absorbed"), (1, 16, 16, 64, 400, 0, 20, "absorbed"), (1, 16, 16, 64, 400, 300, 16, "per head"),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,dim,vdim,rank,piece,front,rows,form", CASES)
def test_form_of_a_portion(heads, dim, vdim, rank, piece, front, rows, form, dtype, monkeypatch):
    cfg = P.config([P.layer(lat(heads, dim, vdim, rank), None)])
    model, w = P.build(cfg, dtype, max_seq=front + rows + 8, max_rows=piece)
    eng = model._ensure_engine()
    kv = eng.new_kv(1, front + rows + 8)
    toks = P.tokens_for(cfg, front + rows, seed=rows)
    ref = P.O.forward(cfg, w, toks)[0][front:]
    got = {}
    for name, env in (("rule", None), ("absorbed", "100000"), ("per head", "1")):
        monkeypatch.setenv("B2_LATENT_MATERIALISE_ROWS", "100000")
        for at in range(0, front, piece):
            eng.append_tokens(kv, 0, toks[at:min(front, at + piece)], restart=at == 0)
        if env is None:
            monkeypatch.delenv("B2_LATENT_MATERIALISE_ROWS")
        else:
            monkeypatch.setenv("B2_LATENT_MATERIALISE_ROWS", env)
        got[name] = eng.append_tokens(kv, 0, toks[front:], list(range(rows)), restart=front == 0).cpu()
    assert P.close(got["rule"], ref, dtype)
    assert P.close(got["absorbed"], got["per head"], dtype, tight=True)
    other = "absorbed" if form == "per head" else "per head"
    assert torch.equal(got["rule"], got[form]) and not torch.equal(got[form], got[other])
