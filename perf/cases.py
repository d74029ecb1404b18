"""Timed cases of the decoder: what a program that serves a model with this framework has it do, through `dsk.Model`.

Two kinds of models.  DeepSeek shapes (`.dseek` tensors): one token through `forward`, or a short greedy completion through
`decode_greedy`.  Layer-list designs (`config.json` tensors): a prompt through `forward_chunk`, or decoding through `decode_greedy`,
`sample` and `forward`.  Weights are random values of the checkpoint's shapes and types, made on the GPU from the seed, few layers deep
(the layers of a model are alike); the caches hold a context where the case decodes.  `exact` restates every design in float64.
"""
import math
import os
import sys
import zlib

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepseek.cpp_b200"))
import dsk  # noqa: E402

DEV = "cuda:0"
EPS = 1e-5

# layer shapes of the DeepSeek family (K-quants: hidden sizes rounded up to whole blocks of 256)
DEEPSEEK = {
    "v2lite": dict(dim=2048, hidden=10944, heads=16, q_rank=0, experts=64, top=6, ff=1408, shared=2, scale=1.0, groups=1, keep=1, v3=0),
    "v2": dict(dim=5120, hidden=12288, heads=128, q_rank=1536, experts=160, top=6, ff=1536, shared=2, scale=16.0, groups=8, keep=3, v3=0),
    "v3": dict(dim=7168, hidden=18432, heads=128, q_rank=1536, experts=256, top=8, ff=2048, shared=1, scale=2.5, groups=8, keep=4, v3=1),
}
NOPE, ROPE, VDIM, KVR = 128, 64, 128, 512
BLOCK_BYTES = {"q2_k": 84, "q3_k": 110}


def listed():
    return [
        # one token of the largest model that one GPU holds, in the format it is served in: small products behind one another, latency
        dict(name="v2_q2k_token", design="deepseek", shape="v2", quant="q2_k", layers=3, vocab=102400, context=144, greedy=0),
        # a completion of the small model in its 8-bit format, tokens fed back on the device
        dict(name="v2lite_f8_completion", design="deepseek", shape="v2lite", quant="f8e5m2", layers=8, vocab=102400, context=16, greedy=16),
        # the widest layers and the other K-quant
        dict(name="v3_q3k_token", design="deepseek", shape="v3", quant="q3_k", layers=2, vocab=129280, context=40, greedy=0),
        # prompts in one call: recurrence, latent attention and routed experts; windowed, latent and recurrent mixers with a shared expert
        layer_list("desarax_prompt_2048", "Desarax", "sa", 2048, prompt=2048, chunk=2048, wanted=64, vocab=4096, ff=1408),
        layer_list("netusun_prompt_2048", "Netusun", "aml", 2048, prompt=2048, chunk=2048, wanted=64, vocab=4096, ff=1408),
        # a prompt of ragged length, cut into steps by the engine; only the last token's logits over a whole vocabulary are wanted
        layer_list("rutulix_prompt_1500", "Rutulix", "aa", 2048, prompt=1500, chunk=512, wanted=1, vocab=102400, ff=8192),
        # a middle-sized model, every size of the prompt odd, most rows scored
        layer_list("nalizen_prompt_777", "Nalizen", "ra", 1024, prompt=777, chunk=777, wanted=300, vocab=2000, ff=768),
        # 32-bit matrices
        layer_list("zetivik_fp32_prompt_600", "Zetivik", "pl", 1024, quant="fp32", prompt=600, chunk=1024, wanted=16, vocab=8000, ff=2816),
        # the smallest portion that a prompt comes in: latency
        layer_list("rutulix_portion_45", "Rutulix", "aa", 1024, prompt=45, chunk=256, wanted=1, vocab=32000, ff=4096),
        # decoding behind a context: routed experts and carried state; dense layers with two mixers
        layer_list("desarax_decode", "Desarax", "sasa", 2048, context=700, greedy=15, vocab=102400, ff=1408),
        layer_list("zetivik_decode", "Zetivik", "plpl", 2048, context=700, greedy=15, vocab=102400, ff=5632),
        # a whole short answer: a few tokens in, greedy tokens out
        layer_list("netusun_answer", "Netusun", "amal", 2048, prompt=3, chunk=256, greedy=24, wanted=1, vocab=102400, ff=1408),
    ]


def layer_list(name, design, pattern, width, *, ff, vocab, quant="bf16", prompt=0, chunk=256, wanted=0, context=0, greedy=0, window=0, experts=64, top=6):
    """pattern: one letter a layer, as in the bench's sizes.  context > 0: a state that already holds that many tokens, and every pass
    decodes `greedy` + 1 tokens more; else a pass is a new sequence of `prompt` tokens with `wanted` rows of logits, then `greedy` tokens."""
    c = dict(design=design, pattern=pattern, width=width, ff=ff, vocab=vocab, quant=quant, prompt=prompt, chunk=chunk, wanted=wanted, context=context,
             greedy=greedy, window=window or width // 2, experts=experts, top=top)
    return dict(name=name, **c) if name else c


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["deepseek", "prompt", "prompt", "decode"])
    if kind == "deepseek":
        shape = rng.choice(["v2lite", "v2lite", "v2"])
        quant = rng.choice(["q2_k", "q3_k", "f8e5m2", "fp16"] if shape == "v2lite" else ["q2_k", "q3_k"])
        return dict(design="deepseek", shape=shape, quant=quant, layers=rng.randint(2, 3), vocab=256 * rng.randint(40, 400), context=log(1, 150),
                    greedy=rng.randint(0, 12) if quant in ("f8e5m2", "fp16") else 0)
    width = rng.choice([768, 1024, 1024, 1280, 2048])
    if kind == "decode":
        design, pattern = rng.choice([("Desarax", "sa"), ("Zetivik", "pl"), ("Zetivik", "lp"), ("Rutulix", "aa"), ("Nalizen", "ra")])
        return layer_list("", design, pattern, width, ff=8 * log(32, 176), vocab=rng.randint(4000, 60000), context=log(20, 700), greedy=rng.randint(3, 16),
                          window=rng.randint(100, 1024), experts=rng.choice([8, 16, 64]), top=rng.randint(1, 6))
    design, pattern = rng.choice([("Desarax", "sa"), ("Desarax", "a"), ("Netusun", "am"), ("Netusun", "ml"), ("Rutulix", "a"), ("Nalizen", "ra"), ("Zetivik", "pl")])
    prompt = log(33, 2048)
    return layer_list("", design, pattern, width, ff=8 * log(32, 176), vocab=rng.randint(1000, 8000), quant=rng.choice(["bf16", "bf16", "bf16", "fp32"]) if prompt < 700 else "bf16",
                      prompt=prompt, chunk=rng.choice([256, 512, 2048]), wanted=min(prompt, rng.randint(16, 100)), window=rng.randint(64, 1024),
                      experts=rng.choice([8, 16, 64]), top=rng.randint(1, 6))


# ---- weights: every tensor from the seed and its name ----------------------------------------------------------------------
def normal(seed, name, shape, scale=1.0, base=0.0):
    g = torch.Generator(device=DEV).manual_seed(zlib.crc32(f"{seed}/{name}".encode()))
    return torch.randn(shape, device=DEV, generator=g).mul_(scale).add_(base)


def uniform(seed, name, shape, lo, hi):
    g = torch.Generator(device=DEV).manual_seed(zlib.crc32(f"{seed}/{name}".encode()))
    return torch.rand(shape, device=DEV, generator=g).mul_(hi - lo).add_(lo)


def token_ids(case, seed, n):
    return np.random.RandomState(seed % (1 << 31)).randint(0, case["vocab"], n).astype(np.int32)


# ---- DeepSeek shapes ----------------------------------------------------------------------------------------------------------
def ds_shape(case):
    z = dict(DEEPSEEK[case["shape"]])
    if case["quant"] in BLOCK_BYTES:
        for k in ("hidden", "ff"):
            z[k] = (z[k] + 255) // 256 * 256
    return z


def ds_tensors(case):
    """(matrices: name -> (rows, columns, experts or 0), fp32 vectors: name -> shape)."""
    z = ds_shape(case)
    mats = {"model.embed": (case["vocab"], z["dim"], 0), "model.output": (case["vocab"], z["dim"], 0)}
    vecs = {"model.norm.weight": (z["dim"],)}
    for l in range(case["layers"]):
        p = f"model.layers.{l}."
        vecs[p + "attn.norm.weight"] = vecs[p + "mlp.norm.weight"] = (z["dim"],)
        vecs[p + "attn.kv_a_norm.weight"] = (KVR,)
        if z["q_rank"]:
            vecs[p + "attn.q_a_norm.weight"] = (z["q_rank"],)
            mats[p + "attn.wq_a"] = (z["q_rank"], z["dim"], 0)
            mats[p + "attn.wq_b"] = (z["heads"] * (NOPE + ROPE), z["q_rank"], 0)
        else:
            mats[p + "attn.wq"] = (z["heads"] * (NOPE + ROPE), z["dim"], 0)
        mats[p + "attn.wkv_a"] = (KVR + ROPE, z["dim"], 0)
        mats[p + "attn.wkv_b"] = (z["heads"] * (NOPE + VDIM), KVR, 0)
        mats[p + "attn.wo"] = (z["dim"], z["heads"] * VDIM, 0)
        if l == 0:
            for n, rc in (("w1", (z["hidden"], z["dim"])), ("w2", (z["dim"], z["hidden"])), ("w3", (z["hidden"], z["dim"]))):
                mats[p + "mlp." + n] = rc + (0,)
            continue
        vecs[p + "moegate.weight"] = (z["experts"], z["dim"])
        if z["v3"]:
            vecs[p + "moegate.bias"] = (z["experts"],)
        for q, f, e in (("mlp.", z["ff"], z["experts"]), ("shared_mlp.", z["shared"] * z["ff"], 0)):
            mats[p + q + "w1"], mats[p + q + "w2"], mats[p + q + "w3"] = (f, z["dim"], e), (z["dim"], f, e), (f, z["dim"], e)
    return mats, vecs


def ds_vector(seed, name, shape):
    if name.endswith("moegate.weight"):
        return normal(seed, name, shape, 4.0 * shape[-1] ** -0.5)
    if name.endswith("moegate.bias"):
        return normal(seed, name, shape, 0.01)
    return normal(seed, name, shape, 0.1, 1.0)


def ds_matrix(case, seed, name, rows, cols, e):
    """Payload of a matrix (of expert e of a stack): (bytes or values, block scales or None)."""
    key, quant = f"{name}#{e}", case["quant"]
    if quant in BLOCK_BYTES:
        g = torch.Generator(device=DEV).manual_seed(zlib.crc32(f"{seed}/{key}".encode()))
        q = torch.randint(0, 256, (rows, cols // 256, BLOCK_BYTES[quant]), dtype=torch.uint8, device=DEV, generator=g)
        d = np.float16(0.1 / math.sqrt(cols))
        put = lambda at, v: q[..., at:at + 2].copy_(torch.from_numpy(np.frombuffer(np.float16(v).tobytes(), np.uint8).copy()).to(DEV))  # noqa: E731
        if quant == "q2_k":
            put(80, d), put(82, d * 1.5)
        else:
            put(108, d / 8)
        return q.reshape(rows, -1), None
    x = normal(seed, key, (rows, cols), 1.0 if name == "model.embed" else cols ** -0.5)
    if quant == "fp16":
        return x.half(), None
    R, C = -(-rows // 128), -(-cols // 128)
    xp = torch.zeros(R * 128, C * 128, device=DEV)
    xp[:rows, :cols] = x
    blk = xp.view(R, 128, C, 128)
    scale = 57344.0 / blk.abs().amax(dim=(1, 3)).clamp(min=1e-12)
    q = (blk * scale[:, None, :, None]).clamp(-57344.0, 57344.0).to(torch.float8_e5m2).view(torch.uint8)
    return q.reshape(R * 128, C * 128)[:rows, :cols].contiguous(), scale.reciprocal()


def ds_model(case, seed):
    z, c = ds_shape(case), dsk.Config()
    c.dim, c.hidden_dim, c.n_layers, c.n_heads, c.vocab_size, c.max_seq_len = z["dim"], z["hidden"], case["layers"], z["heads"], case["vocab"], 1024
    c.rope_theta, c.norm_eps, c.act_silu, c.first_k_dense_replace = 10000.0, 1e-6, 1, 1
    c.n_shared_experts, c.n_routed_experts, c.n_active_routed, c.moe_intermediate_size = z["shared"], z["experts"], z["top"], z["ff"]
    c.routed_scaling_factor, c.n_group, c.topk_group, c.topk_method = z["scale"], z["groups"], z["keep"], 1 if z["groups"] > 1 else 0
    c.norm_topk_prob = c.scoring_sigmoid = c.is_v3 = z["v3"]
    c.kv_lora_rank, c.q_lora_rank, c.qk_nope_head_dim, c.qk_rope_head_dim, c.v_head_dim = KVR, z["q_rank"], NOPE, ROPE, VDIM
    c.quant, c.original_max_position = dsk.QUANT_IDS[case["quant"]], 4096
    c.bs0, c.bs1 = (128, 128) if case["quant"] == "f8e5m2" else (0, 0)
    m = dsk.Model(c, device=0)
    mats, vecs = ds_tensors(case)
    for name, shape in vecs.items():
        t = ds_vector(seed, name, shape)
        m.upload_device(name, "F32", shape, t.data_ptr(), t.numel() * 4)
    kind = {"q2_k": "U8", "q3_k": "U8", "f8e5m2": "F8_E5M2", "fp16": "F16"}[case["quant"]]
    for name, (rows, cols, ne) in mats.items():
        parts = [ds_matrix(case, seed, name, rows, cols, e) for e in range(max(1, ne))]
        q = torch.stack([p[0] for p in parts]) if ne else parts[0][0]
        torch.cuda.synchronize()
        m.upload_device(name + ".weight", kind, tuple(q.shape), q.data_ptr(), q.numel() * q.element_size())
        if parts[0][1] is not None:
            s = torch.stack([p[1] for p in parts]) if ne else parts[0][1]
            torch.cuda.synchronize()
            m.upload_device(name + ".scale", "F32", tuple(s.shape), s.data_ptr(), s.numel() * 4)
    m.finalize()
    return m


# ---- layer-list designs --------------------------------------------------------------------------------------------------------
def ll_config(case):
    W, win, d = case["width"], case["window"], case["design"]
    hd = 128 if W >= 2048 else 64
    H = W // hd
    G = H // 4 if H % 4 == 0 else H
    rank, moe = W // 4, dict(experts=case["experts"], top=case["top"])
    layers = []
    for i, ch in enumerate(case["pattern"]):
        if d == "Desarax":
            ff = {"kind": "moe", "router": dict(moe, scale=1.0), "expert": {"ff": case["ff"], "limit": 7.0}}
            if ch == "s":
                layers.append({"type": "mamba2", "mlp": ff, "mixer": {"heads": W // 32, "vdim": 64, "state": hd, "groups": 4, "conv": 4, "norm_groups": 4}})
            else:
                layers.append({"type": "latent_attention", "mlp": ff, "mixer": {"heads": H, "dim": hd, "vdim": hd, "kv_rank": rank, "mask": {"size": win}, "scale": hd ** -0.5}})
        elif d == "Rutulix":
            layers.append({"type": "attention", "mlp": {"kind": "dense", "ff": case["ff"]},
                           "mixer": {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": win}, "rot": {"dims": hd // 2, "base": 10000.0}}})
        elif d == "Nalizen":
            if ch == "r":
                layers.append({"type": "hgrn2", "mlp": {"kind": "dense", "ff": 2 * case["ff"]}, "mixer": {"heads": H, "dim": hd, "vdim": hd}})
            else:
                layers.append({"type": "attention", "mlp": {"kind": "moe", "router": moe, "expert": {"ff": case["ff"]}},
                               "mixer": {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": win}, "rot": {"dims": hd // 2, "base": 500000.0}}})
        elif d == "Zetivik":
            if ch == "p":
                left = {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": win}, "rot": {"dims": hd, "base": 500000.0}}
                right = {"heads": H, "kv_heads": H // 2, "dim": hd, "vdim": hd, "conv": 4}
                layers.append({"type": "parallel", "mlp": {"kind": "dense", "ff": case["ff"], "limit": 7.0},
                               "mixer": {"left": left, "right": right, "left_scale": 0.5, "right_scale": 0.5}})
            else:
                layers.append({"type": "lightning", "mlp": None, "mixer": {"heads": H, "dim": hd, "vdim": hd, "decay": [1.0 - 2.0 ** (-1.0 - 8.0 * h / H) for h in range(H)]}})
        else:
            ff = {"kind": "dense", "ff": 3 * case["ff"]} if i == 0 else \
                 {"kind": "moe", "router": dict(moe, scale=2.5, groups={"count": 4, "keep": 3}), "expert": {"ff": case["ff"]}, "shared": {"ff": 2 * case["ff"]}}
            if ch == "a":
                mx = {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "softcap": 50.0, "mask": {"size": win}, "conv": 4}
            elif ch == "l":
                mx = {"heads": H, "dim": hd, "rot_dim": hd // 2, "vdim": hd, "kv_rank": rank, "q_rank": 3 * W // 8, "scale": (1.5 * hd) ** -0.5,
                      "rot": {"dims": hd // 2, "base": 500000.0}}
            else:
                mx = {"heads": H, "dim": hd, "vdim": hd, "gate_cap": 15.0}
            layers.append({"type": {"a": "attention", "l": "latent_attention", "m": "mlstm"}[ch], "mixer": mx, "mlp": ff})
    cfg = {"architecture": d, "vocab": case["vocab"], "width": W, "layers": layers, "norm": {"eps": EPS}}
    if d == "Desarax":
        cfg.update(residual_mult=0.5, logit_scale=1.0, token_side={"dim": 32})
        cfg["norm"]["groups"] = 4
    if d == "Nalizen":
        cfg.update(embedding={"scale": 2.0}, token_side={"dim": 32})
    if d == "Zetivik":
        cfg["logit_softcap"] = 50.0
    return cfg


def ll_tensors(cfg):
    """name -> (shape, kind of values); a leading expert axis is written "e*"."""
    W, V, d, n = cfg["width"], cfg["vocab"], cfg["architecture"], len(cfg["layers"])
    T = {"embed": ((V, W), "embed"), "final.norm": ((W,), "small" if d == "Zetivik" else "norm")}
    if d == "Rutulix":
        T["head"] = ((V, W), "mat")
    if d == "Nalizen":
        T["final.norm.b"] = ((W,), "small")
    side = (cfg.get("token_side") or {}).get("dim", 0)
    if side:
        T["side.embed"] = ((V, side * n), "embed")
    for i, lc in enumerate(cfg["layers"]):
        p, mx, ff, ty = f"l{i}.", lc["mixer"], lc["mlp"], lc["type"]
        q = p + "mix."
        T[p + "norm1"] = ((W,), "small" if d == "Zetivik" else "norm")
        if ty == "mamba2":
            inner, gn, H = mx["heads"] * mx["vdim"], mx["groups"] * mx["state"], mx["heads"]
            ch = inner + 2 * gn
            T.update({q + "in": ((inner + ch + H, W), "mat"), q + "conv": ((ch, mx["conv"]), "conv"), q + "conv.b": ((ch,), "small"), q + "dt_bias": ((H,), (-3.0, 0.0)),
                      q + "A_log": ((H,), (-0.7, 1.4)), q + "D": ((H,), "norm"), q + "norm": ((inner,), "norm"), q + "o": ((W, inner), "mat")})
        elif ty == "latent_attention" and d == "Desarax":
            H, D, P, R = mx["heads"], mx["dim"], mx["vdim"], mx["kv_rank"]
            T.update({q + "q": ((H * D, W), "mat"), q + "uk": ((H * D, R), "mat"), q + "uv": ((H * P, R), "mat"), q + "o": ((W, H * P), "mat"), q + "dkv": ((R, W), "mat"),
                      q + "dkv.norm": ((R,), "norm")})
        elif ty == "latent_attention":
            H, D, P, R, Q, Rd = mx["heads"], mx["dim"], mx["vdim"], mx["kv_rank"], mx["q_rank"], mx["rot_dim"]
            T.update({q + "dq": ((Q, W), "mat"), q + "dq.norm": ((Q,), "norm"), q + "uq": ((H * (D + Rd), Q), "mat"), q + "dkv": ((R + Rd, W), "mat"), q + "dkv.norm": ((R,), "norm"),
                      q + "uk": ((H * D, R), "mat"), q + "uv": ((H * P, R), "mat"), q + "sink": ((H,), "small"), q + "g": ((H * P, W), "mat"), q + "o": ((W, H * P), "mat")})
        elif ty in ("hgrn2", "lightning", "mlstm"):
            H, D, P = mx["heads"], mx["dim"], mx["vdim"]
            T.update({q + "q": ((H * D, W), "mat"), q + "v": ((H * P, W), "mat"), q + "o": ((W, H * P), "mat")})
            if ty == "hgrn2":
                T.update({q + "f": ((H * D, W), "mat"), q + "f.b": ((H * D,), "small"), q + "lower": ((H * D,), (0.0, 0.9)), q + "norm": ((P,), "norm")})
            else:
                T.update({q + "k": ((H * D, W), "mat"), q + "g": ((H * P, W), "mat"), q + "norm": ((H * P,), "norm")})
            if ty == "mlstm":
                T.update({q + "i": ((H, W), "mat"), q + "i.b": ((H,), "small"), q + "f": ((H, W), "mat"), q + "f.b": ((H,), (1.0, 6.0))})
        elif ty == "parallel":
            a, b, l, r = mx["left"], mx["right"], q + "left.", q + "right."
            H, G, D = a["heads"], a["kv_heads"], a["dim"]
            for t, rows in (("q", H * D), ("k", G * D), ("v", G * D)):
                T.update({l + t: ((rows, W), "mat"), l + t + ".b": ((rows,), "small")})
            T.update({l + "q.norm": ((D,), "norm"), l + "k.norm": ((D,), "norm"), l + "g": ((H, W), "mat"), l + "o": ((W, H * D), "mat")})
            H, G, D, P = b["heads"], b["kv_heads"], b["dim"], b["vdim"]
            for t, rows in (("q", G * D), ("k", G * D), ("v", H * P)):
                T.update({r + t: ((rows, W), "mat"), r + t + ".conv": ((rows, b["conv"]), "conv")})
            T.update({r + "b": ((H, W), "mat"), r + "a": ((H, W), "mat"), r + "A_log": ((H,), (-0.7, 1.4)), r + "dt_bias": ((H,), (-5.0, -1.0)), r + "norm": ((P,), "norm"),
                      r + "g": ((H * P, W), "mat"), r + "o": ((W, H * P), "mat")})
        else:   # grouped-query attention of Rutulix, Nalizen and Netusun
            H, G, D = mx["heads"], mx["kv_heads"], mx["dim"]
            T.update({q + "q": ((H * D, W), "mat"), q + "k": ((G * D, W), "mat"), q + "o": ((W, H * D), "mat")})
            if d == "Rutulix":
                T.update({q + "q.norm": ((H * D,), "norm"), q + "k.norm": ((G * D,), "norm"), q + "talk": ((H, H), "talk")})
            else:
                T[q + "v"] = ((G * D, W), "mat")
            if d == "Nalizen":
                T[q + "g"] = ((H * D, W), "mat")
            if d == "Netusun":
                for t, rows in (("q", H * D), ("k", G * D), ("v", G * D)):
                    T[q + t + ".conv"] = ((rows, mx["conv"]), "conv")
                T.update({q + "q.norm": ((D,), "norm"), q + "k.norm": ((D,), "norm")})
        if d in ("Rutulix", "Netusun"):
            T.update({p + "norm1b": ((W,), "norm"), p + "norm2": ((W,), "norm"), p + "norm2b": ((W,), "norm")})
        if d == "Netusun":
            T.update({p + "ls1": ((W,), "norm"), p + "ls2": ((W,), "norm")})
        if d == "Nalizen":
            T.update({p + "norm1.b": ((W,), "small"), p + "norm2": ((W,), "norm"), p + "norm2.b": ((W,), "small"), p + "shift": ((W,), (0.0, 0.9))})
        if d == "Zetivik" and ff:
            T[p + "norm2"] = ((W,), "small")
        if side:
            T.update({p + "side.gate": ((side, W), "mat"), p + "side.proj": ((W, side), "mat"), p + "side.norm": ((W,), "norm")})
        if not ff:
            continue
        m = p + "mlp."
        if ff["kind"] == "moe":
            E, f = ff["router"]["experts"], ff["expert"]["ff"]
            T.update({m + "router": ((E, W), "router"), m + "e*.up": ((E, f, W), "mat"), m + "e*.down": ((E, W, f), "mat")})
            if d != "Nalizen":
                T[m + "e*.gate"] = ((E, f, W), "mat")
            if d == "Desarax":
                T[m + "correction"] = ((E,), "small")
            if d == "Nalizen":
                T[m + "router.b"] = ((E,), "small")
            if "shared" in ff:
                f = ff["shared"]["ff"]
                T.update({m + "shared.sg": ((1, W), "mat"), m + "shared.gate": ((f, W), "mat"), m + "shared.up": ((f, W), "mat"), m + "shared.down": ((W, f), "mat")})
        else:
            T.update({m + "up": ((ff["ff"], W), "mat"), m + "down": ((W, ff["ff"]), "mat")})
            if d == "Rutulix":
                T.update({m + "up.b": ((ff["ff"],), "small"), m + "down.b": ((W,), "small"), m + "act": ((2,), "small")})
            else:
                T[m + "gate"] = ((ff["ff"], W), "mat")
    return T


def ll_tensor(seed, name, shape, kind):
    if isinstance(kind, tuple):
        t = uniform(seed, name, shape, *kind)
    elif kind == "talk":
        t = torch.eye(shape[0], device=DEV) + normal(seed, name, shape, 0.1)
    else:
        scale = {"mat": shape[-1] ** -0.5, "router": 2.0 * shape[-1] ** -0.5, "embed": 1.0, "conv": 0.5, "norm": 0.1, "small": 0.1}[kind]
        t = normal(seed, name, shape, scale, 1.0 if kind == "norm" else 0.0)
    return t.to(torch.bfloat16)


def ll_model(case, seed):
    cfg = ll_config(case)
    hc, specs = dsk.ARCHITECTURES[case["design"]](cfg, quant=case["quant"], max_seq_len=0 if case["context"] else case["prompt"] + case["greedy"] + 8, chunk=case["chunk"])
    m = dsk.Model(hc, device=0, layers=specs)
    for name, (shape, kind) in ll_tensors(cfg).items():
        t = ll_tensor(seed, name, shape, kind)
        torch.cuda.synchronize()
        for e in range(shape[0] if "*" in name else 1):
            x = t[e] if "*" in name else t
            m.upload_device(name.replace("*", str(e)), "BF16", tuple(x.shape), x.data_ptr(), x.numel() * 2)
    m.finalize()
    return m


# ---- the timed path --------------------------------------------------------------------------------------------------------------
class State:
    """A loaded model with what it holds of a sequence; the model's memory is given back with it."""

    def __init__(self, case, model, tokens):
        self.case, self.model, self.tokens, self.at = case, model, tokens, case["context"]
        self.want = list(range(len(tokens) - case.get("wanted", 0), len(tokens)))

    def __del__(self):
        self.model.close()


def prepare(case, seed):
    if case["design"] == "deepseek":
        s = State(case, ds_model(case, seed), token_ids(case, seed, case["context"] + 1))
        for pos in range(case["context"]):
            s.model.forward(int(s.tokens[pos]), pos, dsk.HYDRATE_KV_CACHE)
        return s
    s = State(case, ll_model(case, seed), token_ids(case, seed, case["context"] or case["prompt"]))
    for at in range(0, case["context"], 4):   # the context came in as decoded tokens do
        last = at + 4 >= case["context"]
        part = s.tokens[at:at + 4]
        s.model.forward_chunk(part, at, [len(part) - 1] if last else [])
    return s


def decode(m, at, greedy):
    """`greedy` tokens on the device, the next one by the sampler, its logits."""
    tokens, _ = m.decode_greedy(at, greedy)
    logits, _ = m.forward(m.sample(0.0), at + greedy)
    return tokens, logits


def run(state):
    c, m = state.case, state.model
    if c["design"] == "deepseek":
        logits, _ = m.forward(int(state.tokens[-1]), c["context"], want_logits=not c["greedy"])
        if not c["greedy"]:
            return {"logits": logits}
        tokens, logits = decode(m, c["context"] + 1, c["greedy"])
        return {"tokens": tokens, "logits": logits}
    if c["context"]:
        tokens, logits = decode(m, state.at, c["greedy"])
        state.at += c["greedy"] + 1
        return {"tokens": tokens, "logits": logits}
    rows = m.forward_chunk(state.tokens, 0, state.want)
    if not c["greedy"]:
        return {"rows": rows}
    tokens, logits = decode(m, c["prompt"], c["greedy"])
    return {"rows": rows, "tokens": tokens, "logits": logits}


# ---- bytes and operations ----------------------------------------------------------------------------------------------------------
def work(case):
    n_out = case["greedy"] + 1
    if case["design"] == "deepseek":
        z = ds_shape(case)
        per = {"q2_k": 84 / 256, "q3_k": 110 / 256, "f8e5m2": 1.0 + 4 / 16384, "fp16": 2.0}[case["quant"]]
        mats, _ = ds_tensors(case)
        elements = sum(r * c * (z["top"] if e else 1) for n, (r, c, e) in mats.items() if n != "model.embed")
        gates = 4.0 * (case["layers"] - 1) * z["experts"] * z["dim"]
        passes = n_out + (1 if case["greedy"] else 0)
        kv = 2.0 * case["layers"] * (case["context"] + passes / 2) * z["heads"] * (NOPE + ROPE + VDIM)
        return {"bytes": passes * (elements * per + gates + kv) + 4.0 * case["vocab"], "flops": passes * (2.0 * elements + gates / 2 + kv)}
    cfg = ll_config(case)
    es = 2 if case["quant"] == "bf16" else 4
    mat, active, att, state = 0.0, 0.0, 0.0, 0.0   # stored matrix elements, those of one token, attention multiply-adds of one visible key, carried floats
    for name, (shape, kind) in ll_tensors(cfg).items():
        if kind in ("mat", "router"):
            n = float(np.prod(shape))
            if name == "head":
                continue
            used = case["top"] / shape[0] if "*" in name else 1.0
            active += n * used
            mat += n * min(1.0, used * max(1, case["prompt"])) if not case["context"] else n * used
    for lc in cfg["layers"]:
        for mx in ([lc["mixer"]["left"], lc["mixer"]["right"]] if lc["type"] == "parallel" else [lc["mixer"]]):
            if "mask" in mx or "rot_dim" in mx:
                att += mx["heads"] * (mx["dim"] + mx["vdim"] + mx.get("rot_dim", 0))
            else:
                state += mx["heads"] * mx.get("dim", mx.get("state", 0)) * mx["vdim"]
    head = float(case["vocab"]) * case["width"]
    flops = nbytes = 0.0
    if not case["context"]:
        T = case["prompt"]
        keys = min(T, case["window"]) / 2.0
        flops += 2.0 * T * (active + att * keys + 2 * state) + 2.0 * head * case["wanted"]
        nbytes += es * (mat + head) + 4.0 * (2 * T * case["width"] + case["wanted"] * case["vocab"])
    if case["context"] or case["greedy"]:
        seen = min(case["window"], case["context"] + case["prompt"])
        flops += 2.0 * n_out * (active + head + att * seen + 2 * state)
        nbytes += n_out * (es * (active + head) + 4.0 * (2 * state + att * seen / 4)) + 4.0 * case["vocab"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["design"] == "deepseek":   # K-quants: a last bit can turn the rounding of an 8-bit activation, and that one the next layer's
        return {"rel": 3e-2, "max": 0.3} if case["quant"] in BLOCK_BYTES else {"rel": 2e-4, "max": 5e-3}
    if case["quant"] == "fp32" or case["context"] or case["prompt"] <= 4:   # fp32 activations throughout
        return {"rel": 2e-4, "max": 5e-3}
    return {"rel": 3e-2 if case["design"] in ("Desarax", "Netusun", "Nalizen") else 1e-2, "max": 0.99 if case["design"] in ("Desarax", "Netusun", "Nalizen") else 0.2}


# ---- float64 -----------------------------------------------------------------------------------------------------------------------
def rms(x, eps, groups=1):
    g = x.reshape(*x.shape[:-1], groups, -1)
    return (g / (g.square().mean(-1, keepdim=True) + eps).sqrt()).reshape(x.shape)


def layer_norm(x, w, b=0.0):
    d = x - x.mean(-1, keepdim=True)
    return d / (d.square().mean(-1, keepdim=True) + EPS).sqrt() * w + b


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


silu, sigmoid = torch.nn.functional.silu, torch.sigmoid


def rotate(x, dims, base, pairs):
    """x [tokens, heads, dim]: the first `dims` entries turn by position, entries (2i, 2i + 1) or (i, i + dims / 2) together; angles are 32-bit products."""
    i = torch.arange(dims // 2, device=DEV, dtype=torch.float64)
    f = (base ** (-2.0 * i / dims)).float()
    a = (torch.arange(x.shape[0], device=DEV).float()[:, None] * f).double()[:, None, :]
    r = x[..., :dims]
    u, w = (r[..., 0::2], r[..., 1::2]) if pairs else (r[..., :dims // 2], r[..., dims // 2:])
    c, s = a.cos(), a.sin()
    y = torch.stack((u * c - w * s, w * c + u * s), -1).reshape(r.shape) if pairs else torch.cat((u * c - w * s, w * c + u * s), -1)
    return torch.cat((y, x[..., dims:]), -1)


def attend(q, k, v, scale, seen, cap=0.0, sink=None, talk=None):
    """q [T, H, D] against k [T, G, D], v [T, G, P]; seen [T, T]; sink [H]: a score in the denominator that has no value."""
    rep = q.shape[1] // k.shape[1]
    s = scale * torch.einsum("thd,jhd->htj", q, k.repeat_interleave(rep, 1))
    if talk is not None:
        s = torch.einsum("gh,htj->gtj", talk, s)
    if cap:
        s = cap * torch.tanh(s / cap)
    s = s.masked_fill(~seen, -math.inf)
    if sink is not None:
        s = torch.cat((s, sink[:, None, None].expand(-1, s.shape[1], 1)), -1)
    p = s.softmax(-1)
    return torch.einsum("htj,jhp->thp", p[..., :v.shape[0]], v.repeat_interleave(rep, 1))


def causal_conv(x, w):
    taps = w.shape[1]
    xp = torch.cat((x.new_zeros(taps - 1, x.shape[1]), x))
    return sum(xp[j:j + x.shape[0]] * w[:, j] for j in range(taps))


class Exact64:
    """A layer-list model in float64 over a whole sequence at once (recurrences token by token)."""

    def __init__(self, case, seed):
        self.case, self.cfg, self.seed = case, ll_config(case), seed
        self.shapes, self.held = ll_tensors(self.cfg), {}

    def w(self, name, e=None):
        if name not in self.held:   # kept as stored
            self.held[name] = ll_tensor(self.seed, name, *self.shapes[name])
        t = self.held[name]
        return (t if e is None else t[e]).double()

    def mm(self, x, name, e=None):
        return x @ self.w(name, e).T

    def moe(self, p, ff, x):
        d, top, E = self.cfg["architecture"], ff["router"]["top"], ff["router"]["experts"]
        z = self.mm(x, p + "router")
        if d == "Desarax":
            s = sigmoid(z)
            pick = (s + self.w(p + "correction")).topk(top, -1).indices
            wts = s.gather(-1, pick)
            wts = wts / (wts.sum(-1, keepdim=True) + 1e-20) * ff["router"]["scale"]
        elif d == "Nalizen":
            best = (z + self.w(p + "router.b")).topk(top, -1)
            pick, wts = best.indices, best.values.softmax(-1)
        else:
            s, gr = z.softmax(-1), ff["router"]["groups"]
            g = s.reshape(len(s), gr["count"], -1).amax(-1).topk(gr["keep"], -1).indices
            open_ = torch.zeros(len(s), gr["count"], dtype=torch.bool, device=DEV).scatter_(1, g, True).repeat_interleave(E // gr["count"], 1)
            pick = s.masked_fill(~open_, -1.0).topk(top, -1).indices
            wts = s.gather(-1, pick) * ff["router"]["scale"]
        y = torch.zeros_like(x)
        for e in range(E):
            t, k = (pick == e).nonzero(as_tuple=True)
            if len(t):
                y.index_add_(0, t, wts[t, k][:, None] * self.mm(self.hidden(p + "e*.", x[t], ff["expert"], e), p + "e*.down", e))
        if "shared" in ff:
            y += sigmoid(self.mm(x, p + "shared.sg")) * self.mm(self.hidden(p + "shared.", x, ff["shared"]), p + "shared.down")
        return y

    def hidden(self, p, x, ff, e=None):
        d, u = self.cfg["architecture"], self.mm(x, p + "up", e)
        if d == "Nalizen" and e is not None:
            return u.clamp(min=0.0).square()
        if d == "Rutulix":
            a, z = torch.nn.functional.softplus(self.w(p + "act")), u + self.w(p + "up.b")
            return torch.where(z > 0, a[0] * z * z, (0.5 + a[1]) * (torch.expm1(z.clamp(max=0.0)) - z)) + z / 2
        g = self.mm(x, p + "gate", e)
        if d == "Nalizen":
            return gelu(g) * u
        if d == "Netusun":
            return silu(g) * u
        g, u = g.clamp(max=ff["limit"]), u.clamp(-ff["limit"], ff["limit"])
        return g * sigmoid(1.702 * g) * (u + 1.0)

    def feed_forward(self, p, ff, x):
        if ff["kind"] == "moe":
            return self.moe(p, ff, x)
        y = self.mm(self.hidden(p, x, ff), p + "down")
        return y + self.w(p + "down.b") if self.cfg["architecture"] == "Rutulix" else y

    def seen(self, n, size):
        i = torch.arange(n, device=DEV)
        if size is None:
            return i[:, None] >= i
        if self.cfg["architecture"] in ("Rutulix", "Zetivik"):
            return (i[:, None] >= i) & (i[:, None] // size == i // size)
        return (i[:, None] >= i) & (i[:, None] - i < size)

    def ssd(self, p, mx, h):
        H, P, N, G, T = mx["heads"], mx["vdim"], mx["state"], mx["groups"], len(h)
        inner, gn = H * P, G * N
        z, xbc, dt = self.mm(h, p + "in").split((inner, inner + 2 * gn, H), 1)
        xbc = silu(causal_conv(xbc, self.w(p + "conv")) + self.w(p + "conv.b"))
        xs, B, C = xbc[:, :inner].reshape(T, H, P), xbc[:, inner:inner + gn].reshape(T, G, N), xbc[:, inner + gn:].reshape(T, G, N)
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias"))
        decay = (-self.w(p + "A_log").exp() * dt).exp()
        B, C = B.repeat_interleave(H // G, 1), C.repeat_interleave(H // G, 1)
        S, y = h.new_zeros(H, N, P), []
        for t in range(T):
            S = decay[t, :, None, None] * S + (dt[t, :, None] * B[t])[:, :, None] * xs[t][:, None, :]
            y.append((S * C[t][:, :, None]).sum(1))
        y = (torch.stack(y) + self.w(p + "D")[:, None] * xs).reshape(T, inner)
        return self.mm(rms(y * silu(z), EPS, mx["norm_groups"]) * self.w(p + "norm"), p + "o")

    def latent(self, p, mx, h):
        T, H, D, P, R = len(h), mx["heads"], mx["dim"], mx["vdim"], mx["kv_rank"]
        if self.cfg["architecture"] == "Desarax":
            c = rms(self.mm(h, p + "dkv"), EPS) * self.w(p + "dkv.norm")
            o = attend(self.mm(h, p + "q").reshape(T, H, D), self.mm(c, p + "uk").reshape(T, H, D), self.mm(c, p + "uv").reshape(T, H, P), mx["scale"], self.seen(T, mx["mask"]["size"]))
            return self.mm(o.reshape(T, -1), p + "o")
        rot, Rd = mx["rot"], mx["rot_dim"]
        q = self.mm(rms(self.mm(h, p + "dq"), EPS) * self.w(p + "dq.norm"), p + "uq").reshape(T, H, D + Rd)
        d = self.mm(h, p + "dkv")
        c = rms(d[:, :R], EPS) * self.w(p + "dkv.norm")
        turn = lambda v: rotate(v, rot["dims"], rot["base"], False)  # noqa: E731
        q = torch.cat((q[..., :D], turn(q[..., D:])), -1)
        k = torch.cat((self.mm(c, p + "uk").reshape(T, H, D), turn(d[:, None, R:]).expand(-1, H, -1)), -1)
        o = attend(q, k, self.mm(c, p + "uv").reshape(T, H, P), mx["scale"], self.seen(T, None), sink=self.w(p + "sink"))
        return self.mm(sigmoid(self.mm(h, p + "g")) * o.reshape(T, -1), p + "o")

    def attention(self, p, mx, h):
        d, T, H, G, D = self.cfg["architecture"], len(h), mx["heads"], mx["kv_heads"], mx["dim"]
        q, k = self.mm(h, p + "q"), self.mm(h, p + "k")
        seen, rot = self.seen(T, mx["mask"]["size"]), mx.get("rot")
        if d == "Rutulix":
            v, q, k = k.reshape(T, G, D), rms(q, EPS) * self.w(p + "q.norm"), rms(k, EPS) * self.w(p + "k.norm")
            q, k = (rotate(z.reshape(T, -1, D), rot["dims"], rot["base"], True) for z in (q, k))
            o = attend(q, k, v, mx["scale"], seen, talk=self.w(p + "talk"))
        elif d == "Nalizen":
            q, k = (rms(rotate(z.reshape(T, -1, D), rot["dims"], rot["base"], False), EPS) for z in (q, k))
            o = attend(q, k, self.mm(h, p + "v").reshape(T, G, D), mx["scale"], seen).reshape(T, -1) * sigmoid(self.mm(h, p + "g"))
        elif d == "Netusun":
            q, k, v = (causal_conv(z, self.w(p + n + ".conv")).reshape(T, -1, D) for n, z in (("q", q), ("k", k), ("v", self.mm(h, p + "v"))))
            o = attend(rms(q, EPS) * self.w(p + "q.norm"), rms(k, EPS) * self.w(p + "k.norm"), v, mx["scale"], seen, cap=mx["softcap"], sink=h.new_zeros(H))
        else:
            q, k = ((z + self.w(p + n + ".b")).reshape(T, -1, D) for n, z in (("q", q), ("k", k)))
            v = (self.mm(h, p + "v") + self.w(p + "v.b")).reshape(T, G, D)
            q, k = (rotate(rms(z, EPS) * self.w(p + n + ".norm"), rot["dims"], rot["base"], False) for n, z in (("q", q), ("k", k)))
            o = attend(q, k, v, mx["scale"], seen) * sigmoid(self.mm(h, p + "g"))[..., None]
        return self.mm(o.reshape(T, -1), p + "o")

    def delta(self, p, mx, h):
        T, H, G, D, P = len(h), mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"]
        q, k, v = (silu(causal_conv(self.mm(h, p + n), self.w(p + n + ".conv"))) for n in "qkv")
        unit = lambda z: z / (z.square().sum(-1, keepdim=True) + 1e-6).sqrt()  # noqa: E731
        q, k = unit(q.reshape(T, G, D)) / math.sqrt(D), unit(k.reshape(T, G, D))
        q, k, v = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1), v.reshape(T, H, P)
        beta = sigmoid(self.mm(h, p + "b"))
        g = (-self.w(p + "A_log").exp() * torch.nn.functional.softplus(self.mm(h, p + "a") + self.w(p + "dt_bias"))).exp()
        S, y = h.new_zeros(H, D, P), []
        for t in range(T):
            S = g[t, :, None, None] * S
            u = beta[t, :, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
            S = S + k[t][:, :, None] * u[:, None, :]
            y.append((S * q[t][:, :, None]).sum(1))
        y = rms(torch.stack(y), EPS) * self.w(p + "norm") * silu(self.mm(h, p + "g")).reshape(T, H, P)
        return self.mm(y.reshape(T, -1), p + "o")

    def linear(self, ty, p, mx, h):
        T, H, D, P = len(h), mx["heads"], mx["dim"], mx["vdim"]
        q, v = self.mm(h, p + "q").reshape(T, H, D), self.mm(h, p + "v").reshape(T, H, P)
        S, y = h.new_zeros(H, D, P), []
        if ty == "hgrn2":
            low = self.w(p + "lower")
            f = (low + (1.0 - low) * sigmoid(self.mm(h, p + "f") + self.w(p + "f.b"))).reshape(T, H, D)
            q = silu(q)
            for t in range(T):
                S = f[t][:, :, None] * S + (1.0 - f[t])[:, :, None] * v[t][:, None, :]
                y.append((S * q[t][:, :, None]).sum(1))
            return self.mm((rms(torch.stack(y), EPS) * self.w(p + "norm")).reshape(T, -1), p + "o")
        k, gate = self.mm(h, p + "k").reshape(T, H, D), sigmoid(self.mm(h, p + "g"))
        if ty == "lightning":
            q, k, v = silu(q), silu(k), silu(v)
            a = torch.tensor(mx["decay"], device=DEV, dtype=torch.float32).double()[:, None, None]
            for t in range(T):
                S = a * S + k[t][:, :, None] * v[t][:, None, :]
                y.append((S * q[t][:, :, None]).sum(1))
            return self.mm(rms(torch.stack(y).reshape(T, -1), EPS) * self.w(p + "norm") * gate, p + "o")
        cap, q = mx["gate_cap"], q / math.sqrt(D)
        li = cap * torch.tanh((self.mm(h, p + "i") + self.w(p + "i.b")) / cap)
        lf = torch.nn.functional.logsigmoid(cap * torch.tanh((self.mm(h, p + "f") + self.w(p + "f.b")) / cap))
        n, m = h.new_zeros(H, D), h.new_zeros(H)
        for t in range(T):
            new = torch.maximum(lf[t] + m, li[t])
            keep, write, m = (lf[t] + m - new).exp(), (li[t] - new).exp(), new
            S = keep[:, None, None] * S + (write[:, None] * k[t])[:, :, None] * v[t][:, None, :]
            n = keep[:, None] * n + write[:, None] * k[t]
            y.append((S * q[t][:, :, None]).sum(1) / (torch.maximum((n * q[t]).sum(-1).abs(), (-m).exp()) + 1e-6)[:, None])
        return self.mm(rms(torch.stack(y), EPS).reshape(T, -1) * self.w(p + "norm") * gate, p + "o")

    def mixer(self, ty, p, mx, h):
        if ty == "mamba2":
            return self.ssd(p, mx, h)
        if ty == "latent_attention":
            return self.latent(p, mx, h)
        if ty == "parallel":
            return mx["left_scale"] * self.attention(p + "left.", mx["left"], h) + mx["right_scale"] * self.delta(p + "right.", mx["right"], h)
        return self.attention(p, mx, h) if ty == "attention" else self.linear(ty, p, mx, h)

    def logits(self, tokens, rows):
        cfg, d = self.cfg, self.cfg["architecture"]
        tok = torch.as_tensor(np.asarray(tokens), device=DEV, dtype=torch.long)
        x = self.w("embed")[tok] * (cfg.get("embedding") or {}).get("scale", 1.0)
        mult, side = cfg.get("residual_mult", 1.0), (cfg.get("token_side") or {}).get("dim", 0)
        for i, lc in enumerate(cfg["layers"]):
            p, ty, mx, ff = f"l{i}.", lc["type"], lc["mixer"], lc["mlp"]
            w = lambda n: self.w(p + n)  # noqa: E731, B023
            mix = lambda h: self.mixer(ty, p + "mix.", mx, h)  # noqa: E731, B023
            ffn = lambda h: self.feed_forward(p + "mlp.", ff, h)  # noqa: E731, B023
            if d == "Desarax":
                h = rms(x, EPS, cfg["norm"]["groups"]) * w("norm1")
                x = x + mult * (mix(h) + ffn(h))
            elif d == "Rutulix":
                x = x + layer_norm(mix(layer_norm(x, w("norm1"))), w("norm1b"))
                x = x + layer_norm(ffn(layer_norm(x, w("norm2"))), w("norm2b"))
            elif d == "Nalizen":
                before = torch.cat((torch.zeros_like(x[:1]), x[:-1]))
                x = x + layer_norm(mix(x + (before - x) * w("shift")), w("norm1"), w("norm1.b"))
                x = x + layer_norm(ffn(x), w("norm2"), w("norm2.b"))
            elif d == "Zetivik":
                x = x + mix(rms(x, EPS) * (1.0 + w("norm1")))
                if ff:
                    x = x + ffn(rms(x, EPS) * (1.0 + w("norm2")))
            else:
                x = x + w("ls1") * (rms(mix(rms(x, EPS) * w("norm1")), EPS) * w("norm1b"))
                x = x + w("ls2") * (rms(ffn(rms(x, EPS) * w("norm2")), EPS) * w("norm2b"))
            if side:
                row = self.w("side.embed")[tok, i * side:(i + 1) * side]
                x = x + mult * rms(self.mm(gelu(self.mm(x, p + "side.gate")) * row, p + "side.proj"), EPS) * w("side.norm")
        x = x[rows]
        if d in ("Rutulix", "Nalizen"):
            x = layer_norm(x, self.w("final.norm"), self.w("final.norm.b") if d == "Nalizen" else 0.0)
        else:
            x = rms(x, EPS, cfg["norm"].get("groups", 1)) * ((1.0 if d == "Zetivik" else 0.0) + self.w("final.norm"))
        z = self.mm(x, "head" if d == "Rutulix" else "embed") * cfg.get("logit_scale", 1.0)
        cap = cfg.get("logit_softcap")
        return cap * torch.tanh(z / cap) if cap else z


def halves(b):
    return b.contiguous().view(torch.float16).double()


def dequantised(case, seed, name, rows, cols, e=0):
    """A DeepSeek matrix in float64."""
    q, s = ds_matrix(case, seed, name, rows, cols, e)
    quant = case["quant"]
    if quant == "fp16":
        return q.double()
    if quant == "f8e5m2":
        return q.view(torch.float8_e5m2).double() * s.double().repeat_interleave(128, 0)[:rows].repeat_interleave(128, 1)[:, :cols]
    b = q.reshape(-1, BLOCK_BYTES[quant])
    shift = torch.tensor([0, 2, 4, 6], device=DEV, dtype=torch.uint8)[:, None]
    low = lambda qs: ((qs.reshape(-1, 2, 1, 32) >> shift) & 3).reshape(-1, 16, 16).double()  # noqa: E731  (128 values in four shifts of 32 bytes)
    if quant == "q2_k":
        sc = b[:, :16]
        x = halves(b[:, 80:82])[:, :, None] * (sc & 15).double()[:, :, None] * low(b[:, 16:80]) - (halves(b[:, 82:84]) * (sc >> 4).double())[:, :, None]
        return x.reshape(rows, cols)
    mask, sc = b[:, :32], b[:, 96:108]   # high bits: bit (128-half x 4 + shift step) of byte l; scales: 4 low bits each, then 2 high bits each
    bit = torch.arange(8, device=DEV, dtype=torch.uint8)[:, None]
    high = ((mask[:, None, :] >> bit) & 1).reshape(-1, 16, 16).double()
    lo4 = torch.cat((sc[:, :8] & 15, sc[:, :8] >> 4), 1)
    hi2 = torch.cat([(sc[:, 8:12] >> s_) & 3 for s_ in (0, 2, 4, 6)], 1)
    scale = (lo4 | (hi2 << 4)).double() - 32.0
    return (halves(b[:, 108:110])[:, :, None] * scale[:, :, None] * (low(b[:, 32:96]) - 4.0 * (1.0 - high))).reshape(rows, cols)


def eight_bit(case, x):
    """What a K-quant product reads of its activations: blocks of 256 as 8-bit numbers with a scale.  Other types: the activations."""
    if case["quant"] not in BLOCK_BYTES:
        return x
    b = x.reshape(*x.shape[:-1], -1, 256)
    top = b.gather(-1, b.abs().argmax(-1, keepdim=True))
    v = torch.where(top == 0, torch.zeros_like(b), (b * (-127.0 / torch.where(top == 0, 1.0, top))).round().clamp(max=127.0))
    return (v * top * (-1.0 / 127.0)).reshape(x.shape)


class ExactDeepSeek:
    """A DeepSeek model in float64; keys and values are rounded to the cache's 16 bits, K-quant activations to their 8."""

    def __init__(self, case, seed):
        self.case, self.seed, self.z = case, seed, ds_shape(case)
        self.mats, self.vecs = ds_tensors(case)

    def vec(self, name):
        return ds_vector(self.seed, name, self.vecs[name]).double()

    def mm(self, x, name, e=0):
        rows, cols, _ = self.mats[name]
        return eight_bit(self.case, x) @ dequantised(self.case, self.seed, name, rows, cols, e).T

    def norm(self, x, name):
        return rms(x, 1e-6) * self.vec(name)

    def turn(self, x):
        """Rotary positions of the last ROPE entries: interleaved in place (v3), or gathered to halves."""
        T = x.shape[0]
        f = 1.0 / (10000.0 ** (torch.arange(0, ROPE, 2, device=DEV, dtype=torch.float32) / ROPE))
        a = (torch.arange(T, device=DEV).float()[:, None] * f).double()[:, None, :]
        u, w = x[..., 0::2], x[..., 1::2]
        u, w = u * a.cos() - w * a.sin(), u * a.sin() + w * a.cos()
        return torch.stack((u, w), -1).reshape(x.shape) if self.z["v3"] else torch.cat((u, w), -1)

    def gate(self, p, h):
        z, E = self.z, self.z["experts"]
        s = h @ self.vec(p + "moegate.weight").T
        s = sigmoid(s) + self.vec(p + "moegate.bias") if z["v3"] else s.softmax(-1)
        pool = s
        if z["groups"] > 1:   # the best `keep` of every group stand back
            g = s.reshape(len(s), z["groups"], -1)
            g = g.scatter(-1, g.topk(z["keep"], -1).indices, -math.inf)
            pool = torch.where(torch.isinf(g), s.reshape(g.shape), torch.full_like(g, -math.inf)).reshape(len(s), E)
        pick = pool.topk(z["top"], -1).indices
        wts = s.gather(-1, pick)
        return pick, (wts / wts.sum(-1, keepdim=True) if z["v3"] else wts) * z["scale"]

    def mlp(self, p, h, e=0):
        return self.mm(silu(self.mm(h, p + "w1", e)) * self.mm(h, p + "w3", e), p + "w2", e)

    def logits(self, tokens, rows):
        z, T, H = self.z, len(tokens), self.z["heads"]
        tok = torch.as_tensor(np.asarray(tokens), device=DEV, dtype=torch.long)
        x = dequantised(self.case, self.seed, "model.embed", self.case["vocab"], z["dim"])[tok]
        i = torch.arange(T, device=DEV)
        for l in range(self.case["layers"]):
            p = f"model.layers.{l}."
            a = p + "attn."
            h = self.norm(x, a + "norm.weight")
            q = self.mm(self.norm(self.mm(h, a + "wq_a"), a + "q_a_norm.weight"), a + "wq_b") if z["q_rank"] else self.mm(h, a + "wq")
            q = q.reshape(T, H, NOPE + ROPE)
            q = torch.cat((q[..., :NOPE], self.turn(q[..., NOPE:])), -1)
            c = self.mm(h, a + "wkv_a")
            kv = self.mm(self.norm(c[:, :KVR], a + "kv_a_norm.weight"), a + "wkv_b").reshape(T, H, NOPE + VDIM)
            k = torch.cat((kv[..., :NOPE], self.turn(c[:, None, KVR:]).expand(-1, H, -1)), -1).half().double()
            o = attend(q, k, kv[..., NOPE:].half().double(), (NOPE + ROPE) ** -0.5, i[:, None] >= i)
            x = x + self.mm(o.reshape(T, -1), a + "wo")
            h = self.norm(x, p + "mlp.norm.weight")
            if l == 0:
                x = x + self.mlp(p + "mlp.", h)
                continue
            pick, wts = self.gate(p, h)
            y = self.mlp(p + "shared_mlp.", h)
            for e in pick.unique().tolist():
                t, k_ = (pick == e).nonzero(as_tuple=True)
                y.index_add_(0, t, wts[t, k_][:, None] * self.mlp(p + "mlp.", h[t], e))
            x = x + y
        return self.mm(self.norm(x[rows], "model.norm.weight"), "model.output")


def exact(case, seed):
    deepseek = case["design"] == "deepseek"
    m = (ExactDeepSeek if deepseek else Exact64)(case, seed)
    seq = list(token_ids(case, seed, case["context"] + 1 if deepseek else case["context"] or case["prompt"]))
    wanted = case.get("wanted") or 1
    rows = m.logits(seq, list(range(len(seq) - wanted, len(seq))))
    if deepseek and not case["greedy"]:
        return {"logits": rows[0]}
    if not case["greedy"]:
        return {"rows": rows}
    out = {} if deepseek or case["context"] else {"rows": rows}
    last = rows[-1:]
    for _ in range(case["greedy"] + 1):
        seq.append(int(last.argmax()))
        last = m.logits(seq, [len(seq) - 1])
    return {**out, "tokens": None, "logits": last[0]}
