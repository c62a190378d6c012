"""Timed cases: the calls that a program built on this package makes, over the sizes that it makes them with.

Two engines are covered through the package's public classes. `Engine` is LLaVA: the vision tower with the projector, prompts of the
7B-wide decoder, and decode steps of one and of many requests. `SeqEngine` runs the layer-list decoders: prompts through single layers
(window attention, gated linear attention, latent attention with experts), a state-space / RWKV pair in true fp32, and decode steps
of a four-layer model. Weights are random of the initialisation that the tests and the benchmark use; decode steps are fed given
tokens, so that their logits do not hang on a near tie of an earlier selection.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "llava-plus-codebase_b200"))

from llava import _b2  # noqa: E402
from llava.model import KatadraConfig, PefivikConfig, SofopelConfig  # noqa: E402

DEV = "cuda"
VOCAB = 32000
PATCHES = 576        # feature rows of a 336-pixel image


# ------------------------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # one picture of a chat turn through vision tower and projector: small products, bound by latency
        {"name": "image", "kind": "encode", "images": 1},
        # an evaluation batch of pictures
        {"name": "images", "kind": "encode", "images": 16},
        # the prompt of a chat turn with a picture (576 feature rows and 128 tokens) through two decoder layers of the 7B width
        {"name": "llama_prompt", "kind": "llama_prompt", "layers": 2, "batch": 1, "tokens": 704},
        # one user's answer: a prompt and the decode steps behind it, 7B width
        {"name": "llama_decode", "kind": "llama_decode", "layers": 4, "batch": 1, "tokens": 704, "steps": 32},
        # a server's batch of 32 answers in step
        {"name": "llama_decode_batch", "kind": "llama_decode", "layers": 2, "batch": 32, "tokens": 96, "steps": 24},
        # a long prompt through one layer of window attention with a gated feed-forward
        {"name": "window_prompt", "kind": "layers", "model": "window", "width": 2048, "tokens": 2048, "f32": False},
        # a ragged prompt through one layer of gated linear attention with a gated feed-forward
        {"name": "gla_prompt", "kind": "layers", "model": "gla", "width": 2048, "tokens": 1900, "f32": False},
        # a prompt through one layer of latent attention with a mixture of experts
        {"name": "latent_prompt", "kind": "layers", "model": "latent", "width": 2048, "tokens": 1536, "f32": False},
        # a short question to a whole four-layer model: latency and launches
        {"name": "short_prompt", "kind": "layers", "model": "mixed", "width": 2048, "tokens": 41, "f32": False},
        # true fp32 (the option for checking a model): a state-space layer and a layer of attention beside RWKV
        {"name": "pair_f32", "kind": "layers", "model": "pair", "width": 1024, "tokens": 600, "f32": True},
        # one user's answer on a four-layer model
        {"name": "mixed_decode", "kind": "layers_decode", "model": "mixed", "width": 2048, "slots": 1, "tokens": 500, "steps": 48},
        # eight users' answers in step, prompts of different length
        {"name": "mixed_decode_batch", "kind": "layers_decode", "model": "mixed", "width": 2048, "slots": 8, "tokens": 160, "steps": 48},
    ]


def log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["encode", "llama_prompt", "llama_decode", "layers", "layers", "layers", "layers_decode", "layers_decode"])
    if kind == "encode":
        return {"kind": kind, "images": rng.randint(1, 16)}
    if kind == "llama_prompt":
        return {"kind": kind, "layers": rng.randint(1, 2), "batch": rng.randint(1, 3), "tokens": log_between(rng, 24, 704)}
    if kind == "llama_decode":
        batch = log_between(rng, 1, 32)
        return {"kind": kind, "layers": 2, "batch": batch, "tokens": log_between(rng, 16, 704 if batch <= 4 else 96), "steps": rng.randint(8, 24)}
    if kind == "layers":
        model = rng.choice(["window", "gla", "latent", "mixed", "pair"])
        f32 = rng.random() < (0.5 if model == "pair" else 0.15)
        top = 600 if f32 else 1200 if model == "mixed" else 2048
        return {"kind": kind, "model": model, "width": rng.choice([768, 1024, 1536] if f32 else [1024, 1280, 1536, 2048]),
                "tokens": log_between(rng, 12, top), "f32": f32}
    return {"kind": kind, "model": rng.choice(["mixed", "gla", "window"]), "width": rng.choice([1024, 1536, 2048]),
            "slots": rng.randint(1, 8), "tokens": log_between(rng, 16, 500), "steps": rng.randint(16, 48)}


# ------------------------------------------------------------------------------------------------------------------ sizes
VIT = "model.vision_tower.vision_tower.vision_model."


def llava_desc(case):
    """A vision tower in front of a token decoder for the picture cases, a decoder behind a token vision tower for the others."""
    d = dict(image_size=336, patch_size=14, vit_hidden=1024, vit_inter=4096, vit_layers=24, vit_heads=16, vit_select_layer=-2, vit_ln_eps=1e-5,
             hidden=4096, inter=256, layers=1, heads=32, vocab=64, rms_eps=1e-5, rope_theta=10000.0, max_batch=1, max_seq=16, max_images=1)
    if case["kind"] == "encode":
        d.update(max_images=case["images"])
    else:
        d.update(image_size=28, vit_hidden=256, vit_inter=256, vit_layers=1, vit_heads=4, vit_select_layer=-1, inter=11008, layers=case["layers"],
                 vocab=VOCAB, max_batch=case["batch"], max_seq=case["tokens"] + case.get("steps", 0) + 8)
    return d


def llava_shapes(d):
    """name -> (shape, kind): w Linear weight, b bias, g norm weight, e embedding."""
    h, I, D, DI, ps = d["hidden"], d["inter"], d["vit_hidden"], d["vit_inter"], d["patch_size"]
    T = (d["image_size"] // ps) ** 2 + 1
    s = {VIT + "embeddings.class_embedding": ((D,), "e"), VIT + "embeddings.patch_embedding.weight": ((D, 3, ps, ps), "w"),
         VIT + "embeddings.position_embedding.weight": ((T, D), "e"), VIT + "pre_layrnorm.weight": ((D,), "g"), VIT + "pre_layrnorm.bias": ((D,), "b")}
    for i in range(d["vit_layers"] + 1 + d["vit_select_layer"]):
        p = VIT + f"encoder.layers.{i}."
        for n in ("q_proj", "k_proj", "v_proj", "out_proj"):
            s[p + f"self_attn.{n}.weight"], s[p + f"self_attn.{n}.bias"] = ((D, D), "w"), ((D,), "b")
        s[p + "mlp.fc1.weight"], s[p + "mlp.fc1.bias"] = ((DI, D), "w"), ((DI,), "b")
        s[p + "mlp.fc2.weight"], s[p + "mlp.fc2.bias"] = ((D, DI), "w"), ((D,), "b")
        for n in ("layer_norm1", "layer_norm2"):
            s[p + n + ".weight"], s[p + n + ".bias"] = ((D,), "g"), ((D,), "b")
    s["model.mm_projector.0.weight"], s["model.mm_projector.0.bias"] = ((h, D), "w"), ((h,), "b")
    s["model.mm_projector.2.weight"], s["model.mm_projector.2.bias"] = ((h, h), "w"), ((h,), "b")
    s["model.embed_tokens.weight"] = ((d["vocab"], h), "e")
    for i in range(d["layers"]):
        p = f"model.layers.{i}."
        for n in ("q_proj", "k_proj", "v_proj", "o_proj"):
            s[p + f"self_attn.{n}.weight"] = ((h, h), "w")
        s[p + "mlp.gate_proj.weight"] = s[p + "mlp.up_proj.weight"] = ((I, h), "w")
        s[p + "mlp.down_proj.weight"] = ((h, I), "w")
        s[p + "input_layernorm.weight"] = s[p + "post_attention_layernorm.weight"] = ((h,), "g")
    s["model.norm.weight"], s["lm_head.weight"] = ((h,), "g"), ((d["vocab"], h), "w")
    return s


def llava_weights(d, gen):
    w = {}
    for k, (shape, kind) in llava_shapes(d).items():
        t = torch.randn(shape, generator=gen, device=DEV, dtype=torch.bfloat16)
        if kind == "w":
            t *= 1.0 / math.sqrt(math.prod(shape[1:]))
        elif kind == "e":
            t *= 1.0 if len(shape) == 2 else 0.5
        elif kind == "b":
            t *= 0.05
        else:
            t = 1.0 + 0.1 * t
        w[k] = t
    return w


def list_config(case):
    """config.json of a layer-list model: the benchmark's layers at the case's width, masks of half the longest prompt."""
    W, name = case["width"], case["model"]
    heads, kv = W // 128, max(1, W // 512)
    while heads % kv:
        kv -= 1
    mlp = {"kind": "dense", "ff": 5 * W // 2, "limit": 7.0}
    rot = {"base": 10000.0, "dims": 128, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    win = {"type": "attention_2", "mlp": mlp, "mixer": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "mask": {"size": 1024, "keep_first": 4},
                                                        "rot": rot, "scale": 128 ** -0.5}}
    dif = {"type": "attention", "mlp": mlp, "mixer": {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 128, "conv": 4, "diff": 0.8, "mask": {"size": 1024},
                                                      "rot": {"base": 1.0e6, "dims": 64}, "scale": 64 ** -0.5}}
    gla = {"type": "gla", "mlp": mlp, "mixer": {"heads": W // 256, "dim": 128, "vdim": 256, "tau": 16.0}}
    if name in ("window", "gla", "mixed"):
        layers = {"window": [win], "gla": [gla], "mixed": [win, dif, gla, win]}[name]
        return {"architecture": "Sofopel", "width": W, "vocab": VOCAB, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0}, "residual_mult": 0.5, "layers": layers}
    if name == "latent":
        moe = {"kind": "moe", "expert": {"ff": W // 4}, "shared": {"ff": W // 2},
               "router": {"experts": 16, "top": 2, "groups": {"count": 4, "keep": 2}, "scale": 2.0}}
        lat = {"type": "latent_attention", "mlp": moe, "mixer": {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5}}
        return {"architecture": "Pefivik", "width": W, "vocab": VOCAB, "norm": {"eps": 1e-5}, "residual_mult": 0.8, "logit_softcap": 25.0, "layers": [lat]}
    mamba = {"type": "mamba2", "mlp": None, "mixer": {"heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}
    par = {"type": "parallel", "mlp": {"kind": "dense", "ff": 4 * W},
           "mixer": {"left": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "bias_max": 2048, "scale": 128 ** -0.5, "softcap": 30.0,
                              "q_temp": {"coef": 0.5, "every": 256}, "rel_rows": 32},
                     "right": {"heads": W // 64, "dim": 64, "decay_rank": 64}, "left_scale": 1.0, "right_scale": 1.0}}
    return {"architecture": "Katadra", "width": W, "vocab": VOCAB, "norm": {"eps": 1e-5}, "layers": [mamba, par]}


CONFIGS = {"Sofopel": SofopelConfig, "Pefivik": PefivikConfig, "Katadra": KatadraConfig}
GLA_RANK = 16


def list_weights(cfg, gen):
    """Tensors of a checkpoint of this configuration, values representable in bfloat16."""
    W, w = cfg["width"], {}

    def lin(o, i, gain=1.0):
        return torch.randn(o, i, generator=gen, device=DEV, dtype=torch.bfloat16) * (gain / math.sqrt(i))

    def vec(n, mean, std):
        return mean + std * torch.randn(n, generator=gen, device=DEV, dtype=torch.bfloat16)

    def uni(n, lo, hi):
        return (lo + (hi - lo) * torch.rand(n, generator=gen, device=DEV)).bfloat16()

    w["embed"], w["head"] = lin(VOCAB, W, math.sqrt(W)), lin(VOCAB, W)
    arch = cfg["architecture"]
    one = 1 if arch == "Pefivik" else W    # that design's norms have one number as weight
    w["final.norm"] = vec(one, 1.0, 0.1)
    if arch == "Katadra":
        w["final.norm.b"] = vec(W, 0.0, 0.1)
    for i, layer in enumerate(cfg["layers"]):
        p, m, t, mlp = f"l{i}.mix.", layer["mixer"], layer["type"], layer["mlp"]
        w[f"l{i}.norm1"] = vec(one, 1.0, 0.1)
        if arch == "Katadra":
            w[f"l{i}.norm1.b"] = vec(W, 0.0, 0.1)
        if mlp and arch != "Sofopel":
            w[f"l{i}.norm2"] = vec(one, 1.0, 0.1)
            if arch == "Katadra":
                w[f"l{i}.norm2.b"] = vec(W, 0.0, 0.1)
        if t in ("attention", "attention_2"):
            H, G, dk, dv, maps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], 2 if t == "attention" else 1
            w[p + "q"], w[p + "k"], w[p + "v"], w[p + "o"] = lin(maps * H * dk, W), lin(maps * G * dk, W), lin(G * dv, W), lin(W, H * dv)
            if maps == 2:
                for n in ("lq1", "lk1", "lq2", "lk2"):
                    w[p + n] = vec(dk, 0.0, 0.1)
                for n, c in (("q", 2 * H * dk), ("k", 2 * G * dk), ("v", G * dv)):
                    w[p + n + ".conv"] = 0.5 * torch.randn(c, m["conv"], generator=gen, device=DEV, dtype=torch.bfloat16)
            else:
                w[p + "g"], w[p + "q.norm"], w[p + "k.norm"] = lin(H, W), vec(dk, 1.0, 0.2), vec(dk, 1.0, 0.2)
        elif t == "gla":
            H, dk, dv = m["heads"], m["dim"], m["vdim"]
            w[p + "q"], w[p + "k"], w[p + "v"], w[p + "g"], w[p + "o"] = lin(H * dk, W), lin(H * dk, W), lin(H * dv, W), lin(H * dv, W), lin(W, H * dv)
            w[p + "a1"], w[p + "a2"], w[p + "a2.b"], w[p + "norm"] = lin(GLA_RANK, W), lin(H * dk, GLA_RANK), uni(H * dk, -1.0, 5.0), vec(dv, 1.0, 0.2)
        elif t == "latent_attention":
            H, dk, dv, r = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
            w[p + "q"], w[p + "dkv"], w[p + "dkv.norm"], w[p + "uk"], w[p + "uv"] = lin(H * dk, W), lin(r, W), uni(r, 0.7, 1.3), lin(H * dk, r), lin(H * dv, r)
            w[p + "sink"], w[p + "g"], w[p + "o"] = vec(H, 0.0, 1.0), lin(H, W), lin(W, H * dv)
        elif t == "mamba2":
            inner, ch, H = m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"], m["heads"]
            w[p + "in"] = lin(inner + ch + H, W)
            w[p + "conv"] = 0.5 * torch.randn(ch, m["conv"], generator=gen, device=DEV, dtype=torch.bfloat16)
            w[p + "conv.b"], w[p + "dt_bias"], w[p + "A_log"], w[p + "D"] = vec(ch, 0.0, 0.1), vec(H, 0.0, 0.5), vec(H, 0.0, 0.5), vec(H, 0.0, 1.0)
            w[p + "norm"], w[p + "o"] = vec(inner, 1.0, 0.1), lin(W, inner)
        else:
            a, r = m["left"], m["right"]
            H, G, dk, dv, n = a["heads"], a["kv_heads"], a["dim"], a["vdim"], r["heads"] * r["dim"]
            q = p + "left."
            w[q + "q"], w[q + "k"], w[q + "v"], w[q + "g"], w[q + "o"] = lin(H * dk, W), lin(G * dk, W), lin(G * dv, W), lin(H * dv, W), lin(W, H * dv)
            w[q + "rel"] = torch.randn(a["rel_rows"], H, generator=gen, device=DEV, dtype=torch.bfloat16)
            q = p + "right."
            for s in "rkvgw":
                w[q + "mu." + s] = uni(W, 0.0, 1.0)
            for s in "rkvg":
                w[q + s] = lin(n, W)
            w[q + "w1"], w[q + "w2"], w[q + "w0"] = lin(r["decay_rank"], W), lin(n, r["decay_rank"]), vec(n, -1.0, 0.5)
            w[q + "u"], w[q + "norm"], w[q + "o"] = 0.5 * torch.randn(r["heads"], r["dim"], generator=gen, device=DEV, dtype=torch.bfloat16), vec(n, 1.0, 0.1), lin(W, n)
        if not mlp:
            continue
        p = f"l{i}.mlp."
        if mlp["kind"] == "moe":
            E, ff, sf = mlp["router"]["experts"], mlp["expert"]["ff"], mlp["shared"]["ff"]
            w[p + "router"] = lin(E, W, 3.0)
            for e in range(E):
                w[p + f"e{e}.gate"], w[p + f"e{e}.up"], w[p + f"e{e}.down"] = lin(ff, W), lin(ff, W), lin(W, ff)
            w[p + "shared.gate"], w[p + "shared.up"], w[p + "shared.down"] = lin(sf, W), lin(sf, W), lin(W, sf)
        else:
            ff = mlp["ff"]
            w[p + "up"], w[p + "down"] = lin(ff, W), lin(W, ff)
            if arch == "Sofopel":
                w[p + "gate"] = lin(ff, W)
    return w


def prompts_of(case, gen):
    """Token ids of every slot: the first has the case's length, further ones are shorter by odd amounts."""
    n = case["tokens"]
    return [torch.randint(0, VOCAB, (max(2, n - 13 * b * n // 160),), generator=gen).tolist() for b in range(case.get("slots", 1))]


# ------------------------------------------------------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    gen, host = torch.Generator(device=DEV).manual_seed(seed), torch.Generator().manual_seed(seed)
    kind = case["kind"]
    if kind in ("encode", "llama_prompt", "llama_decode"):
        d = llava_desc(case)
        eng = _b2.Engine(d, DEV)
        for k, t in llava_weights(d, gen).items():
            eng.set_weight(k, t)
        eng.finalize()
        if kind == "encode":
            return {"kind": kind, "eng": eng, "pixels": torch.randn(case["images"], 3, 336, 336, generator=gen, device=DEV, dtype=torch.bfloat16)}
        B, S = case["batch"], case["tokens"]
        src, feats = llama_inputs(case, gen)
        s = {"kind": kind, "eng": eng, "kv": eng.new_kv(B, d["max_seq"]), "B": B, "S": S, "src": src, "feats": feats}
        if kind == "llama_decode":
            s["fed"] = list(torch.randint(0, VOCAB, (case["steps"], B), generator=gen, device=DEV, dtype=torch.int32))
        return s
    cfg = list_config(case)
    w = list_weights(cfg, gen)
    conf = CONFIGS[cfg["architecture"]](**cfg)
    slots, n = case.get("slots", 1), case["tokens"]
    desc = dict(width=conf.width, vocab=conf.vocab, compute=_b2.COMPUTE_F32 if case.get("f32") else _b2.COMPUTE_BF16, norm_eps=conf.norm_eps, max_batch=slots,
                max_rows=max(n, slots), **conf.model_desc())
    eng = _b2.SeqEngine(desc, conf.layer_descs({k: tuple(t.shape) for k, t in w.items()}), DEV)
    for k, t in w.items():
        eng.set_weight(k, t)
    eng.finalize()
    s = {"kind": kind, "eng": eng, "kv": eng.new_kv(slots, n + case.get("steps", 0) + 8), "prompts": prompts_of(case, host)}
    if kind == "layers_decode":
        s["fed"] = list(torch.randint(0, VOCAB, (case["steps"], slots), generator=gen, device=DEV, dtype=torch.int32))
    return s


def llama_inputs(case, gen):
    """Source index of the prompt rows (token ids; -(row) - 1 for a picture's feature rows) and the feature rows, if the prompt holds them."""
    B, S = case["batch"], case["tokens"]
    src = torch.randint(0, VOCAB, (B, S), generator=gen, device=DEV, dtype=torch.int32)
    if S < PATCHES + 64:
        return src, None
    feats = torch.randn(B * PATCHES, 4096, generator=gen, device=DEV, dtype=torch.bfloat16)
    src[:, 35:35 + PATCHES] = -torch.arange(B * PATCHES, device=DEV, dtype=torch.int32).view(B, PATCHES) - 1
    return src, feats


def run(state):
    eng, kind = state["eng"], state["kind"]
    if kind == "encode":
        return eng.encode_images(state["pixels"])
    kv = state["kv"]
    if kind in ("llama_prompt", "llama_decode"):
        kv.reset()
        logits = eng.prefill(kv, eng.splice(state["src"], state["feats"], state["B"], state["S"]))
        return logits if kind == "llama_prompt" else [logits] + [eng.decode_step(kv, t) for t in state["fed"]]
    if kind == "layers":
        toks = state["prompts"][0]
        logits, residuals = eng.append_tokens(kv, 0, toks, [len(toks) - 1], restart=True, residuals=True)
        return [logits, residuals]
    for b, toks in enumerate(state["prompts"]):
        eng.append_tokens(kv, b, toks, restart=True)
    return [eng.decode_step(kv, t) for t in state["fed"]]


# ------------------------------------------------------------------------------------------------------------------ work
def pairs_seen(n, window=None, chunk=None, keep=0):
    """Visible (row, key) pairs of a causal prompt of n tokens."""
    total = 0
    for i in range(n):
        if chunk:
            total += i % chunk + 1
        elif window:
            first = max(0, i - window + 1)
            total += i + 1 - first + min(keep, first)
        else:
            total += i + 1
    return total


def list_layer_work(layer, W, n):
    """(weights used, flops) of one layer over n tokens of one prompt."""
    m, t, mlp = layer["mixer"], layer["type"], layer["mlp"]
    extra = 0
    if t in ("attention", "attention_2"):
        H, G, dk, dv, maps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], 2 if t == "attention" else 1
        p = W * (maps * (H + G) * dk + G * dv + (H if maps == 1 else 0) + H * dv)
        size = m["mask"]["size"]
        seen = pairs_seen(n, chunk=size) if maps == 2 else pairs_seen(n, window=size, keep=m["mask"]["keep_first"])
        extra = 2 * maps * H * seen * (dk + dv)
    elif t == "gla":
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        p = W * (2 * H * dk + 3 * H * dv + GLA_RANK) + GLA_RANK * H * dk
        extra = 5 * n * H * dk * dv
    elif t == "latent_attention":
        H, dk, dv, r = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
        p = W * (H * dk + r + H + H * dv) + r * H * (dk + dv)
        extra = 2 * H * pairs_seen(n) * (dk + dv)
    elif t == "mamba2":
        H, P, N = m["heads"], m["vdim"], m["state"]
        p = W * (3 * H * P + 2 * m["groups"] * N + H)
        extra = 5 * n * H * P * N
    else:
        a, r = m["left"], m["right"]
        H, G, dk, dv, R, d = a["heads"], a["kv_heads"], a["dim"], a["vdim"], r["heads"] * r["dim"], r["dim"]
        p = W * (H * dk + G * (dk + dv) + 2 * H * dv) + W * (5 * R + r["decay_rank"]) + R * r["decay_rank"]
        extra = 2 * H * pairs_seen(n) * (dk + dv) + 6 * n * R * d
    held = p
    if mlp and mlp["kind"] == "moe":
        E, top, ff, sf = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"], mlp["shared"]["ff"]
        p += W * (E + 3 * sf + top * 3 * ff)
        held += W * (E + 3 * sf + min(E, n * top) * 3 * ff)
    elif mlp:
        q = W * mlp["ff"] * (3 if "limit" in mlp else 2)
        p, held = p + q, held + q
    return held, 2 * n * p + extra


def work(case):
    kind = case["kind"]
    if kind == "encode":
        n, T, D, h = case["images"], PATCHES + 1, 1024, 4096
        per = 2 * PATCHES * 588 * D + 23 * (2 * T * 12 * D * D + 4 * T * T * D) + 2 * PATCHES * (D * h + h * h)
        return {"bytes": 2 * (23 * 12 * D * D + 588 * D + D * h + h * h) + n * 2 * (3 * 336 * 336 + PATCHES * h), "flops": n * per}
    if kind in ("llama_prompt", "llama_decode"):
        L, B, S, N, h, I = case["layers"], case["batch"], case["tokens"], case.get("steps", 0), 4096, 11008
        per, head = 4 * h * h + 3 * h * I, VOCAB * h
        seen = B * pairs_seen(S)
        flops = L * (2 * B * S * per + 4 * seen * h) + 2 * B * head
        bts = 2 * (L * per + head) + 2 * B * S * h + 4 * B * VOCAB + L * B * S * h * 4
        for t in range(N):
            flops += L * (2 * B * per + 4 * B * (S + t + 1) * h) + 2 * B * head
            bts += 2 * (L * per + head) + L * B * (S + t + 1) * h * 4 + 4 * B * VOCAB
        return {"bytes": bts, "flops": flops}
    cfg = list_config(case)
    W, e = cfg["width"], 4 if case.get("f32") else 2
    if kind == "layers":
        n = case["tokens"]
        bts, flops = e * (n * W + VOCAB * W) + 4 * VOCAB, 2 * VOCAB * W
        for layer in cfg["layers"]:
            held, f = list_layer_work(layer, W, n)
            bts, flops = bts + e * held + 4 * n * W, flops + f
        return {"bytes": bts, "flops": flops}
    lens = [len(p) for p in prompts_of(case, torch.Generator().manual_seed(0))]
    bts = flops = 0
    for layer in cfg["layers"]:
        for n in lens:
            held, f = list_layer_work(layer, W, n)
            bts, flops = bts + e * held, flops + f
        m, t = layer["mixer"], layer["type"]
        held, f1 = list_layer_work(layer, W, 1)
        state = 8 * m["heads"] * m["dim"] * m["vdim"] if t == "gla" else 0
        for s in range(case["steps"]):
            bts += e * held + len(lens) * state
            flops += len(lens) * f1
            if t != "gla":
                maps = 2 if t == "attention" else 1
                seen = sum(min(n + s + 1, m["mask"]["size"]) for n in lens)
                bts += 4 * seen * m["kv_heads"] * (maps * m["dim"] + m["vdim"])
                flops += 2 * maps * seen * m["heads"] * (m["dim"] + m["vdim"])
    bts += case["steps"] * (e * VOCAB * W + 4 * len(lens) * VOCAB)
    flops += case["steps"] * 2 * len(lens) * VOCAB * W
    return {"bytes": bts, "flops": flops}


def tolerance(case):
    if case.get("f32"):
        return {"rel": 1e-5, "max": 1e-3}
    # bf16 operands of every product (relative rounding 2^-9), through as many layers as the case has
    if case.get("model") == "latent":   # a router's near tie falls the other way on a few rows, which then take another expert
        return {"rel": 2.5e-2, "max": 0.99}
    return {"rel": 2e-2 if case["kind"] == "encode" else 1e-2, "max": 0.5}


# ------------------------------------------------------------------------------------------------------------------ exact values
def unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def layer_norm(x, g, b, eps):
    m = x.mean(-1, keepdim=True)
    return (x - m) / torch.sqrt(((x - m) ** 2).mean(-1, keepdim=True) + eps) * g + b


def heads_of(x, H):
    """[..., T, H * d] -> [..., H, T, d]"""
    return x.unflatten(-1, (H, -1)).transpose(-2, -3)


def softmax_attend(s, seen, v, sink=None):
    """softmax(s) v over the keys that `seen` allows; sink [H]: one more term exp(sink) in the denominator."""
    s = s.masked_fill(~seen, float("-inf"))
    m = s.amax(-1, keepdim=True)
    if sink is not None:
        m = torch.maximum(m, sink.view(-1, 1, 1))
    e = torch.exp(s - m)
    den = e.sum(-1, keepdim=True)
    if sink is not None:
        den = den + torch.exp(sink.view(-1, 1, 1) - m)
    return (e / den) @ v


def causal(n):
    i = torch.arange(n, device=DEV)
    return i[:, None], i[None, :]


def conv_over_time(u, taps):
    n = taps.shape[1]
    pad = torch.cat([u.new_zeros(n - 1, u.shape[1]), u])
    return sum(pad[j:j + u.shape[0]] * taps[:, j] for j in range(n))


def rotary(rot):
    dims, base, sc = rot["dims"], rot["base"], rot.get("scaling")
    i = torch.arange(dims // 2, device=DEV, dtype=torch.float64)
    f = base ** (-2.0 * i / dims)
    if not sc:
        return f, 1.0

    def turn(t):
        return dims * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))

    lo, hi = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def turned(x, rot, half):
    """x [H, T, d], the rotated pairs lead: (2i, 2i + 1), or (i, i + pairs) in the half layout."""
    f, mag = rotary(rot)
    a = torch.arange(x.shape[1], device=DEV, dtype=torch.float64)[:, None] * f
    c, s, n = torch.cos(a) * mag, torch.sin(a) * mag, len(f)
    out = x.clone()
    iu, iv = (slice(0, n), slice(n, 2 * n)) if half else (slice(0, 2 * n, 2), slice(1, 2 * n, 2))
    u, v = x[..., iu], x[..., iv]
    out[..., iu], out[..., iv] = u * c - v * s, v * c + u * s
    return out


def exact_encode(d, w, px):
    D, H, eps, ps = d["vit_hidden"], d["vit_heads"], d["vit_ln_eps"], d["patch_size"]
    F, B = torch.nn.functional, px.shape[0]

    def W(k):
        return w[VIT + k].double()

    cols = F.unfold(px.double(), ps, stride=ps).transpose(1, 2)
    x = torch.cat([W("embeddings.class_embedding").expand(B, 1, D), cols @ W("embeddings.patch_embedding.weight").flatten(1).T], 1)
    x = F.layer_norm(x + W("embeddings.position_embedding.weight"), (D,), W("pre_layrnorm.weight"), W("pre_layrnorm.bias"), eps)
    for i in range(d["vit_layers"] + 1 + d["vit_select_layer"]):
        p = f"encoder.layers.{i}."

        def lin(y, n):
            return F.linear(y, W(p + n + ".weight"), W(p + n + ".bias"))

        y = F.layer_norm(x, (D,), W(p + "layer_norm1.weight"), W(p + "layer_norm1.bias"), eps)
        q, k, v = (heads_of(lin(y, f"self_attn.{n}_proj"), H) for n in "qkv")
        a = torch.softmax(q @ k.transpose(-1, -2) * (D // H) ** -0.5, -1) @ v
        x = x + lin(a.transpose(1, 2).flatten(2), "self_attn.out_proj")
        y = lin(F.layer_norm(x, (D,), W(p + "layer_norm2.weight"), W(p + "layer_norm2.bias"), eps), "mlp.fc1")
        x = x + lin(y * torch.sigmoid(1.702 * y), "mlp.fc2")
    y = F.gelu(F.linear(x[:, 1:], w["model.mm_projector.0.weight"].double(), w["model.mm_projector.0.bias"].double()))
    return F.linear(y, w["model.mm_projector.2.weight"].double(), w["model.mm_projector.2.bias"].double())


def exact_llama(d, w, x):
    """x [S, hidden] of one request -> normed rows in front of the head."""
    h, H, eps = d["hidden"], d["heads"], d["rms_eps"]
    rot = {"dims": h // H, "base": d["rope_theta"]}
    for i in range(d["layers"]):
        p = f"model.layers.{i}."

        def W(k):
            return w[p + k].double()

        y = unit(x, eps) * W("input_layernorm.weight")
        q, k, v = (heads_of(y @ W(f"self_attn.{n}_proj.weight").T, H) for n in "qkv")
        q, k = turned(q, rot, True), turned(k, rot, True)
        r, c = causal(x.shape[0])
        a = softmax_attend(q @ k.transpose(-1, -2) * (h // H) ** -0.5, c <= r, v)
        x = x + a.transpose(0, 1).flatten(1) @ W("self_attn.o_proj.weight").T
        y = unit(x, eps) * W("post_attention_layernorm.weight")
        g = y @ W("mlp.gate_proj.weight").T
        x = x + (g * torch.sigmoid(g) * (y @ W("mlp.up_proj.weight").T)) @ W("mlp.down_proj.weight").T
    return unit(x, eps) * w["model.norm.weight"].double()


def silu(x):
    return x * torch.sigmoid(x)


def ex_window(h, p, m, eps):
    H, G, n = m["heads"], m["kv_heads"], h.shape[0]
    q = turned(unit(heads_of(h @ p["q"].T, H), eps) * p["q.norm"], m["rot"], True)
    k = turned(unit(heads_of(h @ p["k"].T, G), eps) * p["k.norm"], m["rot"], True)
    k, v = (t.repeat_interleave(H // G, 0) for t in (k, heads_of(h @ p["v"].T, G)))
    r, c = causal(n)
    seen = (c <= r) & ((r - c < m["mask"]["size"]) | (c < m["mask"]["keep_first"]))
    a = softmax_attend(q @ k.transpose(-1, -2) * m["scale"], seen, v, torch.zeros(H, device=DEV, dtype=torch.float64))
    return (a.transpose(0, 1) * torch.sigmoid(h @ p["g"].T)[..., None]).flatten(1) @ p["o"].T


def ex_diff(h, p, m, eps):
    H, G, n = m["heads"], m["kv_heads"], h.shape[0]
    q, k, v = (conv_over_time(h @ p[t].T, p[t + ".conv"]) for t in "qkv")
    q, k = (turned(heads_of(t, 2 * g), m["rot"], False).unflatten(0, (g, 2)) for t, g in ((q, H), (k, G)))
    k, v = k.repeat_interleave(H // G, 0), heads_of(v, G).repeat_interleave(H // G, 0)
    r, c = causal(n)
    seen = (c <= r) & (r // m["mask"]["size"] == c // m["mask"]["size"])
    a = [softmax_attend(q[:, j] @ k[:, j].transpose(-1, -2) * m["scale"], seen, v) for j in (0, 1)]
    lam = torch.exp(p["lq1"] @ p["lk1"]) - torch.exp(p["lq2"] @ p["lk2"]) + m["diff"]
    return (unit(a[0] - lam * a[1], eps) * (1.0 - m["diff"])).transpose(0, 1).flatten(1) @ p["o"].T


def scan(decay, k, v, q, bonus=None):
    """S <- decay * S + k v^T, o = S^T q per head, token by token; all [T, H, d]. With a bonus o reads S_(t-1) + bonus k v^T."""
    S = q.new_zeros(q.shape[1], q.shape[2], v.shape[2])
    out = q.new_zeros(q.shape[0], q.shape[1], v.shape[2])
    for t in range(q.shape[0]):
        kv = k[t][:, :, None] * v[t][:, None, :]
        if bonus is None:
            S = decay[t][:, :, None] * S + kv
            out[t] = (q[t][:, :, None] * S).sum(1)
        else:
            out[t] = (q[t][:, :, None] * (S + bonus[:, :, None] * kv)).sum(1)
            S = decay[t][:, :, None] * S + kv
    return out


def ex_gla(h, p, m, eps):
    H, dk = m["heads"], m["dim"]
    q, k, v = (heads_of(h @ p[t].T, H).transpose(0, 1) for t in "qkv")
    z = (h @ p["a1"].T) @ p["a2"].T + p["a2.b"]
    alpha = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).unflatten(-1, (H, dk))
    o = unit(scan(alpha, k, v, q * dk ** -0.5), eps) * p["norm"]
    return (o.flatten(1) * silu(h @ p["g"].T)) @ p["o"].T


def ex_latent(h, p, m, eps):
    H = m["heads"]
    c = unit(h @ p["dkv"].T, eps) * p["dkv.norm"]
    q, k, v = heads_of(h @ p["q"].T, H), heads_of(c @ p["uk"].T, H), heads_of(c @ p["uv"].T, H)
    r, j = causal(h.shape[0])
    a = softmax_attend(q @ k.transpose(-1, -2) * m["scale"], j <= r, v, p["sink"])
    return (a.transpose(0, 1) * torch.sigmoid(h @ p["g"].T)[..., None]).flatten(1) @ p["o"].T


def ex_mamba2(h, p, m, eps):
    H, P, N, G, n = m["heads"], m["vdim"], m["state"], m["groups"], h.shape[0]
    inner, proj = H * P, h @ p["in"].T
    z, xbc, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * G * N], proj[:, 2 * inner + 2 * G * N:]
    c = silu(conv_over_time(xbc, p["conv"]) + p["conv.b"])
    x = c[:, :inner].reshape(n, H, P)
    Bm, Cm = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (c[:, inner:inner + G * N], c[:, inner + G * N:]))
    dt = torch.nn.functional.softplus(dt + p["dt_bias"], threshold=50.0)
    y = scan(torch.exp(-torch.exp(p["A_log"]) * dt)[..., None], Bm, dt[..., None] * x, Cm) + p["D"][:, None] * x
    y = (y.flatten(1) * silu(z)).unflatten(-1, (m["norm_groups"], -1))
    return (unit(y, eps).flatten(1) * p["norm"]) @ p["o"].T


def ex_parallel(h, p, m, eps):
    a, r, n = m["left"], m["right"], h.shape[0]
    L, R = ({k[len(s):]: v for k, v in p.items() if k.startswith(s)} for s in ("left.", "right."))
    H, G = a["heads"], a["kv_heads"]
    pos = torch.arange(n, device=DEV, dtype=torch.float64)
    temp = 1.0 + a["q_temp"]["coef"] * torch.log(torch.floor((pos + 1) / a["q_temp"]["every"]) + 1)
    q, k = unit(heads_of(h @ L["q"].T, H), eps) * temp[:, None], unit(heads_of(h @ L["k"].T, G), eps)
    k, v = (t.repeat_interleave(H // G, 0) for t in (k, heads_of(h @ L["v"].T, G)))
    half, rows = a["rel_rows"] // 2, a["rel_rows"]
    bucket = torch.tensor([d if d < half else min(rows - 1, half + int(math.floor(math.log(d / half) / math.log(a["bias_max"] / half) * (rows - half))))
                           for d in range(n)], device=DEV)
    i, j = causal(n)
    s = a["softcap"] * torch.tanh(q @ k.transpose(-1, -2) * a["scale"] / a["softcap"]) + L["rel"][bucket[(i - j).clamp(min=0)]].permute(2, 0, 1)
    left = (softmax_attend(s, j <= i, v).transpose(0, 1).flatten(1) * torch.sigmoid(h @ L["g"].T)) @ L["o"].T
    prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    mix = {s: h + (prev - h) * R["mu." + s] for s in "rkvgw"}
    q, k, v = ((mix[s] @ R[s].T).unflatten(-1, (r["heads"], -1)) for s in "rkv")
    decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ R["w1"].T) @ R["w2"].T + R["w0"])).unflatten(-1, (r["heads"], -1))
    o = unit(scan(decay, k, v, q, R["u"].reshape(r["heads"], -1)), eps).flatten(1)
    return a_scale(m, "left_scale") * left + a_scale(m, "right_scale") * ((o * R["norm"] * silu(mix["g"] @ R["g"].T)) @ R["o"].T)


def a_scale(m, k):
    return float(m[k])


def ex_moe(h, p, mlp):
    r = mlp["router"]
    E, G = r["experts"], r["groups"]["count"]
    s = torch.sigmoid(h @ p["router"].T)
    gs = s.unflatten(-1, (G, E // G)).topk(2, -1).values.sum(-1)
    alive = torch.zeros_like(gs, dtype=torch.bool).scatter_(1, gs.topk(r["groups"]["keep"], -1).indices, True).repeat_interleave(E // G, 1)
    top = s.masked_fill(~alive, -1.0).topk(r["top"], -1)
    wgt = torch.zeros_like(s).scatter_(1, top.indices, top.values / (top.values.sum(-1, keepdim=True) + 1e-20) * r["scale"])

    def expert(x, n):
        return (silu(x @ p[n + ".gate"].T) * (x @ p[n + ".up"].T)) @ p[n + ".down"].T

    out = expert(h, "shared")
    for e in range(E):
        rows = wgt[:, e].nonzero().flatten()
        out[rows] += wgt[rows, e, None] * expert(h[rows], f"e{e}")
    return out


def ex_clamped(h, p, mlp):
    g, u = (h @ p["gate"].T).clamp(max=mlp["limit"]), (h @ p["up"].T).clamp(-mlp["limit"], mlp["limit"])
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ p["down"].T


EXACT = {"attention_2": ex_window, "attention": ex_diff, "gla": ex_gla, "latent_attention": ex_latent, "mamba2": ex_mamba2, "parallel": ex_parallel}


def exact_list(cfg, w, tokens):
    """Normed rows in front of the head [T, width] and the residual stream after every layer, of one prompt."""
    eps, arch, m = cfg["norm"]["eps"], cfg["architecture"], cfg.get("residual_mult", 1.0)
    x, stream = w["embed"][torch.tensor(tokens, device=DEV)].double(), []
    for i, layer in enumerate(cfg["layers"]):
        mix, mlp = ({k[len(s):]: v.double() for k, v in w.items() if k.startswith(s)} for s in (f"l{i}.mix.", f"l{i}.mlp."))
        n1, n2 = w[f"l{i}.norm1"].double(), w[f"l{i}.norm2"].double() if f"l{i}.norm2" in w else None
        f = EXACT[layer["type"]]
        if arch == "Sofopel":
            u = unit(x, eps) * n1
            x = x + m * (f(u, mix, layer["mixer"], eps) + ex_clamped(u, mlp, layer["mlp"]))
        elif arch == "Pefivik":
            x = x + m * f(unit(x, eps) * n1, mix, layer["mixer"], eps)
            x = x + m * ex_moe(unit(x, eps) * n2, mlp, layer["mlp"])
        else:
            x = x + layer_norm(f(x, mix, layer["mixer"], eps), n1, w[f"l{i}.norm1.b"].double(), eps)
            if layer["mlp"]:
                y = torch.relu(x @ mlp["up"].T) ** 2 @ mlp["down"].T
                x = x + layer_norm(y, n2, w[f"l{i}.norm2.b"].double(), eps)
        stream.append(x)
    g = w["final.norm"].double()
    return layer_norm(x, g, w["final.norm.b"].double(), eps) if arch == "Katadra" else unit(x, eps) * g, torch.stack(stream)


def exact(case, seed):
    gen, host = torch.Generator(device=DEV).manual_seed(seed), torch.Generator().manual_seed(seed)
    kind = case["kind"]
    if kind in ("encode", "llama_prompt", "llama_decode"):
        d = llava_desc(case)
        w = llava_weights(d, gen)
        if kind == "encode":
            px = torch.randn(case["images"], 3, 336, 336, generator=gen, device=DEV, dtype=torch.bfloat16)
            return torch.cat([exact_encode(d, w, px[b:b + 1]) for b in range(case["images"])])
        src, feats = llama_inputs(case, gen)
        fed = torch.randint(0, VOCAB, (case["steps"], case["batch"]), generator=gen, device=DEV, dtype=torch.int32) if kind == "llama_decode" else None
        rows = []
        for b in range(case["batch"]):
            ids = src[b].long()
            x = w["model.embed_tokens.weight"][ids.clamp(min=0)].double()
            if feats is not None:
                x = torch.where((ids < 0)[:, None], feats[(-ids - 1).clamp(min=0)].double(), x)
            if fed is not None:
                x = torch.cat([x, w["model.embed_tokens.weight"][fed[:, b].long()].double()])
            rows.append(exact_llama(d, w, x)[case["tokens"] - 1:])
        logits = torch.stack(rows, 1) @ w["lm_head.weight"].double().T
        return logits[0] if kind == "llama_prompt" else list(logits)
    cfg = list_config(case)
    w = list_weights(cfg, gen)
    prompts = prompts_of(case, host)
    head, cap = w["head"].double(), cfg.get("logit_softcap")
    if kind == "layers":
        z, stream = exact_list(cfg, w, prompts[0])
        logits = z[-1:] @ head.T
        return [cap * torch.tanh(logits / cap) if cap else logits, stream]
    fed = torch.randint(0, VOCAB, (case["steps"], len(prompts)), generator=gen, device=DEV, dtype=torch.int32)
    rows = [exact_list(cfg, w, toks + fed[:, b].tolist())[0][len(toks):] for b, toks in enumerate(prompts)]
    return list(torch.stack(rows, 1) @ head.T)
