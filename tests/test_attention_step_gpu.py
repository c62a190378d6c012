"""Decode steps whose heads the one-launch attention kernel takes (csrc/attention_bias.cu, attn_step_kernel): sizes at its edges, one to six query heads
a key/value head, windows with kept positions, chunks, two maps over shared values, biases and soft-caps, sinks and gates; slots of one key, of fewer
keys than warps, and of more than one pass. True fp32 against the plain oracles."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def win(heads, kv, dim, vdim, mask=None):
    return "Sofopel", {"type": "attention_2", "mlp": None, "mixer": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": vdim, "scale": 0.2, **({"mask": mask} if mask else {}),
                                                                     "rot": {"base": 500.0, "dims": 8}}}


def two_maps(heads, kv, dim, vdim, chunk):
    return "Sofopel", {"type": "attention", "mlp": None, "mixer": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": vdim, "conv": 3, "diff": 0.7, "mask": {"size": chunk},
                                                                   "rot": {"base": 100.0, "dims": 8}, "scale": 0.2}}


def biased(heads, kv, dim, vdim):
    left = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": vdim, "bias_max": 64, "scale": 0.3, "softcap": 5.0, "q_temp": {"coef": 0.5, "every": 16}, "rel_rows": 16}
    return "Katadra", {"type": "parallel", "mlp": {"kind": "dense", "ff": 40}, "mixer": {"left": left, "right": {"heads": 3, "dim": 16, "decay_rank": 8}, "left_scale": 1.0, "right_scale": 1.0}}


def sinks(heads, kv, dim):
    return "Ramosun", {"type": "attention", "mlp": None, "mixer": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": 0.2, "mask": {"size": 100}, "rot": {"base": 50.0, "dims": 8}}}


CASES = {"one_head": win(1, 1, 32, 4), "two": win(4, 2, 64, 128, {"size": 50, "keep_first": 3}), "three": win(3, 1, 96, 36, {"size": 7, "keep_first": 9}), "four": win(16, 4, 128, 128, {"size": 300}),
         "six": win(6, 1, 128, 100), "maps": two_maps(8, 2, 64, 128, 37), "maps_one": two_maps(2, 1, 32, 8, 1), "biased": biased(6, 2, 32, 64), "sinks": sinks(5, 1, 32), "many_groups": win(8, 8, 32, 32)}


@pytest.mark.parametrize("name", list(CASES))
def test_steps_follow_the_oracle(name):
    import llava.model as M

    arch, lay = CASES[name]
    O = importlib.import_module(f"oracle.{arch.lower()}_oracle")
    cfg = {"architecture": arch, "width": 72, "vocab": 150, "norm": {"eps": 1e-5}, "layers": [lay]}
    w = {k: torch.as_tensor(np.asarray(v, np.float32)) for k, v in O.random_weights(cfg, seed=3).items()}
    lengths, steps = [1, 40, 700, 131], 5
    model = getattr(M, arch + "ForCausalLM")(getattr(M, arch + "Config")(**cfg), {k: v.bfloat16() for k, v in w.items()}, dtype=torch.float32, max_batch=4, max_seq=720, max_rows=700)
    eng = model._ensure_engine()
    toks = torch.randint(0, 150, (4, 705), generator=torch.Generator().manual_seed(5))
    for slots in (1, 4):
        kv = eng.new_kv(4, 720)
        which = [2] if slots == 1 else range(4)
        for b, i in enumerate(which):
            eng.append_tokens(kv, b, toks[i, :lengths[i]].tolist(), restart=True)
        got = [eng.decode_step(kv, torch.stack([toks[i, lengths[i] + t] for i in which]).int()).cpu().double() for t in range(steps)]
        for b, i in enumerate(which):
            ref = torch.as_tensor(np.asarray(O.forward(cfg, w if arch == "Katadra" else {k: v.numpy() for k, v in w.items()}, toks[i, :lengths[i] + steps].tolist())), dtype=torch.float64)[lengths[i]:]
            e = torch.stack([g[b] for g in got]) - ref
            # fp32 throughout: rounding of a layer, some 1e-6 of the logits' spread (the families' tests allow the same)
            assert float(((e ** 2).mean(-1).sqrt() / ref.std(-1)).max()) < 2e-4, (name, slots, i)
        kv.close()
