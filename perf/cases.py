"""Workloads of the engine, called the way a serving program calls it: a loaded model, a ragged batch of token runs through
`Model.infer_raw`, the sampling front half behind every decode step, cached prefixes written back into their slots.

Models are a few layers deep at the widths of the shapes this repository benchmarks, so that one pass shows the layers and the
vocabulary head and not only a long repetition; weights are random.  Four model families stand for the engine's paths:

  rwkv6, rwkv7   the RWKV path (f16 weights, token shift, data-dependent decay / delta rule); also with Int8 / NF4 layers and
                 with f32-exact activations
  panupel        gated delta rule, attention over the whole context beside a matrix memory, dense feed-forwards (bf16 weights)
  kemirax        latent attention over a shared cache, routed experts, gated linear attention (bf16 weights)

`call` is "decode" (every sequence continues a cached prefix by `steps` tokens, one per step, the candidates of every step
sampled on the device and the last logits rows read), "prompt" (new sequences, last rows) or "score" (new sequences, a row per
token).
"""
from __future__ import annotations

import json
import math
import random
import struct

import numpy as np
import torch

from ai00_server_b200 import capi, runtime, synth

TOP_K = 128                     # the nucleus sampler's default
HEAD = 64                       # RWKV head size

# RWKV shapes: hidden size, low ranks (v6: token shift, decay; v7: decay, in-context rate, value, gate)
_V6 = {2048: (7168, 32, 64), 2560: (8960, 32, 64), 4096: (14336, 64, 128)}
_V7_RANKS = (96, 96, 64, 320)


def _rwkv(name, family, call, width, layers, batch, tokens, **more):
    c = {"name": name, "family": family, "call": call, "width": width, "layers": layers, "vocab": 65536, "batch": batch, "tokens": tokens,
         "ragged": False, "steps": 0, "chunk": 128, "precision": 0, "quant": "none"}
    c.update(more)
    return c


def _seq(name, family, call, width, batch, tokens, **more):
    c = {"name": name, "family": family, "call": call, "width": width, "layers": 4 if family == "panupel" else 2, "vocab": 32768, "batch": batch,
         "tokens": tokens, "ragged": False, "steps": 0, "chunk": 512, "precision": 0, "quant": "none"}
    c.update(more)
    return c


def listed():
    return [
        # one user reading an answer token by token: 3B widths, batch 1, bound by latency and launches
        _rwkv("v6_decode_b1", "rwkv6", "decode", 2560, 4, 1, 16, steps=16),
        # a full server, 16 slots, 7B widths: the headline decode
        _rwkv("v6_decode_b16", "rwkv6", "decode", 4096, 3, 16, 16, steps=8),
        # the same server with Int8 layers (`quant` of the reload request)
        _rwkv("v6_int8_decode_b16", "rwkv6", "decode", 4096, 3, 16, 16, steps=8, quant="Int8"),
        # f32-exact activations (Bundle::<f32>), a few users
        _rwkv("v6_f32_decode_b4", "rwkv6", "decode", 2560, 4, 4, 16, steps=12, precision=1),
        # RWKV-7 decode, 8 users
        _rwkv("v7_decode_b8", "rwkv7", "decode", 2560, 4, 8, 16, steps=12),
        # time to the first token of one chat message at 7B widths
        _rwkv("v6_prompt_b1", "rwkv6", "prompt", 4096, 3, 1, 100),
        # the embeddings route's shape: many texts of 512 tokens, 3B widths; the state of the first goes back to the host
        _rwkv("v6_prompt_b32", "rwkv6", "prompt", 2560, 4, 32, 512),
        # the `choose` route: a handful of candidate texts of different lengths, one row per token
        _rwkv("v7_score_b6", "rwkv7", "score", 2560, 4, 6, 61, ragged=True),
        # prompts and decode of the config.json families, 16 sequences, 1024 tokens of context
        _seq("panupel_prompt_b16", "panupel", "prompt", 2048, 16, 1024),
        _seq("panupel_decode_b16", "panupel", "decode", 2048, 16, 1024, steps=16),
        # documents of different lengths through latent attention and routed experts
        _seq("kemirax_prompt_b8", "kemirax", "prompt", 2048, 8, 700, ragged=True),
        _seq("kemirax_decode_b16", "kemirax", "decode", 2048, 16, 777, steps=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    """One more case of the same ranges: families, calls, widths, depths, batches, lengths, chunk sizes, precisions."""
    family = rng.choice(["rwkv6", "rwkv6", "rwkv7", "panupel", "kemirax"])
    if family.startswith("rwkv"):
        call = rng.choice(["decode", "decode", "prompt", "prompt", "score"])
        width = 128 * rng.randint(8, 32)
        layers = rng.randint(1, 3) if width > 2560 else rng.randint(1, 4)
        option = rng.choice(["none", "none", "none", "f32", "Int8", "NF4"])
        more = {"precision": 1 if option == "f32" else 0, "quant": option if option in ("Int8", "NF4") else "none", "chunk": rng.choice([64, 128, 128, 256, 512])}
        if call == "decode":
            return {k: v for k, v in _rwkv("", family, call, width, layers, rng.randint(1, 32), rng.randint(1, 24), steps=rng.randint(4, 16), **more).items() if k != "name"}
        if call == "score":
            return {k: v for k, v in _rwkv("", family, call, width, layers, rng.randint(1, 8), rng.randint(5, 90), ragged=True, **more).items() if k != "name"}
        batch = _log_int(rng, 1, 32)
        tokens = _log_int(rng, 9, max(10, min(1500, (16384 * 2560 if not more["precision"] else 4096 * 2560) // (batch * max(width, 1024)))))
        return {k: v for k, v in _rwkv("", family, call, width, layers, batch, tokens, ragged=rng.random() < 0.5, **more).items() if k != "name"}
    call = rng.choice(["decode", "prompt"])
    width = 128 * rng.randint(4, 16)
    more = {"vocab": rng.choice([32000, 32768, 50304]), "chunk": rng.choice([128, 256, 512]), "layers": rng.choice([2, 4]) if family == "panupel" else 2}
    if call == "decode":
        return {k: v for k, v in _seq("", family, call, width, rng.randint(1, 16), _log_int(rng, 8, 1024), steps=rng.randint(8, 16), **more).items() if k != "name"}
    batch = _log_int(rng, 1, 16)
    return {k: v for k, v in _seq("", family, call, width, batch, _log_int(rng, 20, 1024), ragged=rng.random() < 0.5, **more).items() if k != "name"}


# ----------------------------------------------------------------------------------------------------------------------
# models: shapes, random weights, file images
# ----------------------------------------------------------------------------------------------------------------------
def _shape(case):
    W = case["width"]
    if case["family"] == "rwkv6":
        F, Dm, Dd = _V6.get(W, (W * 7 // 2 // 128 * 128, 64 if W >= 4096 else 32, 128 if W >= 4096 else 64))
        return synth.Shape(6, case["layers"], W, F, V=case["vocab"], Dm=Dm, Dd=Dd)
    Dd, Da, Dv, Dg = _V7_RANKS
    return synth.Shape(7, case["layers"], W, 4 * W, V=case["vocab"], Dd=Dd, Da=Da, Dv=Dv, Dg=Dg)


def _dims(case):
    """Sizes of the config.json families at a width, in the proportions of the benchmarked 2048-wide stacks."""
    W = case["width"]
    H = W // 128
    if case["family"] == "panupel":
        G = next(g for g in (4, 3, 2, 1) if H % g == 0)
        return {"W": W, "V": case["vocab"], "H": H, "G": G, "d": 128, "Hm": max(1, H // 2), "m": 128, "ff": W * 11 // 4 // 64 * 64, "conv": 4, "cap": 15.0, "r": 0.6}
    return {"W": W, "V": case["vocab"], "H": H, "dn": 128, "dr": 64, "dv": 128, "rk": W // 4, "rq": W * 3 // 8, "E": 16 if W > 1024 else 8, "I": 2,
            "top": 4 if W > 1024 else 2, "ff": W // 2, "sff": W, "lim": 2.0, "slim": 1.5, "a": 8, "tau": 8.0}


_PN_ROT = {"base": 5e5, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
_KX_ROT = {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
_EPS = 1e-5
_PN_LEFT, _PN_RIGHT = 1.1, 0.8


def _panupel_kinds(case):
    return ["delta", "parallel"] * (case["layers"] // 2)


def _config(case):
    z = _dims(case)
    cfg = {"architecture": case["family"].capitalize(), "norm": {"eps": _EPS}, "vocab": z["V"], "width": z["W"], "layers": []}
    if case["family"] == "panupel":
        cfg["residual_mult"] = z["r"]
        if case["layers"] == 4:
            cfg["loop"] = {"start": 1, "stop": 3, "times": 1}
        for kind in _panupel_kinds(case):
            if kind == "delta":
                mixer = {"heads": z["H"], "kv_heads": z["G"], "dim": z["d"], "vdim": z["d"], "conv": z["conv"]}
            else:
                mixer = {"left": {"heads": z["H"], "kv_heads": z["G"], "dim": z["d"], "vdim": z["d"], "rot": _PN_ROT, "scale": z["d"] ** -0.5},
                         "right": {"heads": z["Hm"], "dim": z["m"], "vdim": z["m"], "gate_cap": z["cap"]}, "left_scale": _PN_LEFT, "right_scale": _PN_RIGHT}
            cfg["layers"].append({"type": kind, "mixer": mixer, "mlp": {"kind": "dense", "ff": z["ff"]}})
    else:
        # the experts sit in the first layer, whose router sees the embedding row itself: two correct implementations then choose
        # the same experts, and the logits can be compared row by row
        cfg["layers"].append({"type": "latent_attention", "mixer": {"heads": z["H"], "dim": z["dn"], "rot_dim": z["dr"], "vdim": z["dv"], "kv_rank": z["rk"],
                              "q_rank": z["rq"], "rot": _KX_ROT, "scale": (z["dn"] + z["dr"]) ** -0.5},
                              "mlp": {"kind": "moe", "router": {"experts": z["E"], "identity": z["I"], "top": z["top"]}, "expert": {"ff": z["ff"], "limit": z["lim"]},
                                      "shared": {"ff": z["sff"], "limit": z["slim"]}}})
        cfg["layers"].append({"type": "gla", "mixer": {"heads": z["H"], "dim": z["dn"], "vdim": z["dv"], "tau": z["tau"]}, "mlp": None})
    return json.dumps(cfg)


def _spec(case):
    """[(name, shape, lo, hi)]: uniform in [lo, hi], or normal with deviation hi where lo is None."""
    if case["family"].startswith("rwkv"):
        return [(n, s, lo, hi) for n, s, lo, hi in synth.tensor_spec(_shape(case))]
    z, out = _dims(case), []
    W, H = z["W"], z["H"]

    def mat(name, n, k, g=1.0):
        out.append((name, (n, k), None, g / math.sqrt(k)))

    def vec(name, n, lo, hi):
        out.append((name, (n,), lo, hi))

    out.append(("embed", (z["V"], W), None, 1.0))
    if case["family"] == "panupel":
        G, d, Hm, m = z["G"], z["d"], z["Hm"], z["m"]
        if case["layers"] == 4:
            mat("loop.in", W, 2 * W)
        for i, kind in enumerate(_panupel_kinds(case)):
            p = "l%d." % i
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                vec(p + n, W, 0.5, 1.5)
            if kind == "delta":
                for n, rows in (("q", G * d), ("k", G * d), ("v", H * d)):
                    mat(p + "mix." + n, rows, W, 2.0)
                    out.append((p + "mix." + n + ".conv", (rows, z["conv"]), None, 0.6))
                mat(p + "mix.b", H, W, 2.0)
                mat(p + "mix.a", H, W, 2.0)
                vec(p + "mix.A_log", H, -4.0, 0.0)
                vec(p + "mix.dt_bias", H, -4.0, 1.0)
                vec(p + "mix.norm", d, 0.5, 1.5)
                mat(p + "mix.g", H * d, W, 2.0)
                mat(p + "mix.o", W, H * d)
            else:
                q = p + "mix.left."
                mat(q + "q", H * d, W)
                mat(q + "k", G * d, W)
                mat(q + "v", G * d, W)
                vec(q + "q.norm", H * d, 0.5, 1.5)
                vec(q + "k.norm", G * d, 0.5, 1.5)
                out.append((q + "sink", (H,), None, 1.0))
                mat(q + "g", H, W, 2.0)
                mat(q + "o", W, H * d)
                q = p + "mix.right."
                mat(q + "q", Hm * m, W, 1.5)
                mat(q + "k", Hm * m, W, 1.5)
                mat(q + "v", Hm * m, W)
                mat(q + "g", Hm * m, W, 2.0)
                vec(q + "norm", Hm * m, 0.5, 1.5)
                mat(q + "i", Hm, W, 2.0)
                mat(q + "f", Hm, W, 2.0)
                vec(q + "i.b", Hm, -3.0, 1.0)
                vec(q + "f.b", Hm, 0.0, 6.0)
                mat(q + "o", W, Hm * m)
            mat(p + "mlp.gate", z["ff"], W, 2.0)
            mat(p + "mlp.up", z["ff"], W, 2.0)
            mat(p + "mlp.down", W, z["ff"])
        vec("final.norm", W, 0.5, 1.5)
    else:
        dn, dr, dv, rk, rq = z["dn"], z["dr"], z["dv"], z["rk"], z["rq"]
        for i in range(2):
            p = "l%d." % i
            out.append((p + "norm1", (), 0.8, 1.2))
            vec(p + "shift", W, 0.0, 1.0)
            for r in ("rg1", "rg2") if i == 0 else ("rg1",):
                mat(p + r, W, W)
                vec(p + r + ".b", W, -0.5, 1.0)
        mat("l0.mix.dq", rq, W)
        vec("l0.mix.dq.norm", rq, 0.5, 1.5)
        mat("l0.mix.uq", H * (dn + dr), rq, 2.0)
        mat("l0.mix.dkv", rk + dr, W, 2.0)
        vec("l0.mix.dkv.norm", rk, 0.5, 1.5)
        mat("l0.mix.uk", H * dn, rk, 2.0)
        mat("l0.mix.uv", H * dv, rk)
        mat("l0.mix.o", W, H * dv)
        mat("l0.mlp.router", z["E"] + z["I"], W, 2.0)
        vec("l0.mlp.correction", z["E"] + z["I"], -0.05, 0.05)
        for e in ["e%d" % j for j in range(z["E"])] + ["shared"]:
            ff = z["sff"] if e == "shared" else z["ff"]
            mat("l0.mlp.%s.gate" % e, ff, W, 2.0)
            mat("l0.mlp.%s.up" % e, ff, W, 2.0)
            mat("l0.mlp.%s.down" % e, W, ff)
        mat("l0.mlp.shared.sg", 1, W)
        for n, rows in (("q", H * dn), ("k", H * dn), ("v", H * dv), ("g", H * dv), ("a1", z["a"])):
            mat("l1.mix." + n, rows, W)
        mat("l1.mix.o", W, H * dv)
        vec("l1.mix.norm", dv, 0.5, 1.5)
        mat("l1.mix.a2", H * dn, z["a"], 2.0)
        vec("l1.mix.a2.b", H * dn, 1.0, 4.0)
        out.append(("final.norm", (), 0.8, 1.2))
    mat("head", z["V"], W)
    return out


def _weights(case, seed):
    """(flat device tensor in file order, {name: view}); f16 for RWKV, bf16 for the others."""
    spec = _spec(case)
    dtype = torch.float16 if case["family"].startswith("rwkv") else torch.bfloat16
    gen = torch.Generator("cuda").manual_seed(1000003 * int(seed) + 17)
    flat = torch.empty(sum(math.prod(s) for _, s, _, _ in spec), dtype=dtype, device="cuda")
    views, at = {}, 0
    for name, shape, lo, hi in spec:
        n = math.prod(shape)
        v = flat[at:at + n]
        if lo is None:
            v.normal_(0.0, hi, generator=gen)
        else:
            v.uniform_(lo, hi, generator=gen)
        views[name] = v.view(shape)
        at += n
    return flat, views


def _image(case, flat, views):
    """The safetensors file the engine loads."""
    head, off = {"__metadata__": {"format": "pt"}}, 0
    for name, v in views.items():
        head[name] = {"dtype": "F16" if flat.dtype == torch.float16 else "BF16", "shape": list(v.shape), "data_offsets": [off, off + 2 * v.numel()]}
        off += 2 * v.numel()
    text = json.dumps(head, separators=(",", ":")).encode()
    text += b" " * (-len(text) % 8)
    img = np.empty(8 + len(text) + off, np.uint8)
    img[:8] = np.frombuffer(struct.pack("<Q", len(text)), np.uint8)
    img[8:8 + len(text)] = np.frombuffer(text, np.uint8)
    torch.from_numpy(img[8 + len(text):]).copy_(flat.view(torch.uint8))
    return img


def _lengths(case):
    B, T = case["batch"], case["tokens"]
    if not case["ragged"]:
        return [T] * B
    share = np.random.default_rng([B, T]).uniform(0.3, 1.0, B)
    return [T] + [max(1, int(round(T * f))) for f in share[1:]]


def _texts(case, seed):
    """Token ids of every sequence: [prefix or prompt] and, for decode, the tokens that follow.  The lengths belong to the case."""
    rng = np.random.default_rng([int(seed), 5])
    B = case["batch"]
    lens = _lengths(case)
    return [rng.integers(1, case["vocab"], n + case["steps"]).astype(np.uint32) for n in lens], lens


# ----------------------------------------------------------------------------------------------------------------------
# what a program holds, and its calls
# ----------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    flat, views = _weights(case, seed)
    img = _image(case, flat, views)
    del flat, views
    torch.cuda.empty_cache()
    texts, lens = _texts(case, seed)
    B, steps = case["batch"], case["steps"]
    kw = {"max_batch": B, "token_chunk_size": case["chunk"], "precision": case["precision"]}
    if case["quant"] != "none":
        kw.update(quant=case["layers"], quant_type=case["quant"])
    if not case["family"].startswith("rwkv"):
        kw.update(config=_config(case), kv_tokens=sum(n + steps for n in lens) + 64 * B)
    m = runtime.Model(img, **kw)
    slots = np.arange(B, dtype=np.int32)
    rows = sum(lens) if case["call"] == "score" else B
    st = {"call": case["call"], "model": m, "slots": slots, "rwkv": case["family"].startswith("rwkv"),
          "logits": torch.empty((rows, case["vocab"]), dtype=torch.float32, pin_memory=True).numpy()}
    one, last = np.ones(B, np.int32), np.full(B, capi.OPTION_LAST, np.int32)
    if case["call"] == "decode":
        for s in slots:
            m.state.reset(int(s))
        m.infer_raw(slots, np.asarray(lens, np.int32), np.concatenate([t[:n] for t, n in zip(texts, lens)]), last, keep_on_device=True)
        st["cached"] = [m.state.read(int(s)) for s in slots]
        st["steps"] = [np.array([t[n + i] for t, n in zip(texts, lens)], np.uint32) for i in range(steps)]
        st["ntok"], st["option"] = one, last
    else:
        st["tokens"], st["ntok"] = np.concatenate(texts), np.asarray(lens, np.int32)
        st["option"] = np.full(B, capi.OPTION_FULL if case["call"] == "score" else capi.OPTION_LAST, np.int32)
    return st


def run(st):
    m, slots = st["model"], st["slots"]
    if st["call"] == "decode":
        for s, item in zip(slots, st["cached"]):
            m.state.write(item, int(s))
        probs = []
        for i, tok in enumerate(st["steps"]):
            if i + 1 < len(st["steps"]):
                m.infer_raw(slots, st["ntok"], tok, st["option"], keep_on_device=True)
            else:
                m.infer_raw(slots, st["ntok"], tok, st["option"], out=st["logits"])
            probs.append(m.sample_topk(slots, top_k=TOP_K)[1])
        return {"logits": st["logits"], "probs": np.stack(probs)}
    for s in slots:
        m.state.reset(int(s))
    m.infer_raw(slots, st["ntok"], st["tokens"], st["option"], out=st["logits"])
    out = {"logits": st["logits"]}
    if st["rwkv"] and st["call"] == "prompt" and len(slots) > 1:
        out["state"] = m.state.back(0)
    return out


# ----------------------------------------------------------------------------------------------------------------------
# work and tolerance
# ----------------------------------------------------------------------------------------------------------------------
def work(case):
    B, T, V, S = case["batch"], case["tokens"], case["vocab"], case["steps"]
    tokens = sum(_lengths(case))
    rows = tokens if case["call"] == "score" else B
    per_w = {"none": 2.0, "Int8": 1.0 + 4 / 128, "NF4": 0.5 + 2 / 64}[case["quant"]]
    W, L = case["width"], case["layers"]
    wbytes = flops_tok = state = cache_tok = attn_tok = 0.0
    if case["family"].startswith("rwkv"):
        for name, shape, _, _ in _spec(case):
            n = math.prod(shape)
            if not name.startswith("blocks."):
                continue
            if len(shape) == 2 and min(shape) > 512 or ("ffn" in name and len(shape) == 2):
                wbytes += per_w * n
            else:
                wbytes += 2.0 * n
            if len(shape) >= 2 and shape[0] != 1 and n > 4 * W:
                flops_tok += 2.0 * n
        state = 4.0 * L * W * (HEAD + 2)                       # f32 state of one sequence
        flops_tok += L * W * HEAD * 8.0
    else:
        z = _dims(case)
        H = z["H"]
        for name, shape, _, _ in _spec(case):
            n = math.prod(shape)
            if name in ("embed", "head"):
                continue
            routed = ".mlp.e" in name
            share = z["top"] / (z["E"] + z["I"]) if routed else 1.0
            seen = min(1.0, share * (B if S else tokens)) if routed else 1.0
            wbytes += 2.0 * n * seen
            if len(shape) == 2:
                flops_tok += 2.0 * n * share
        if case["family"] == "panupel":
            k = L // 2
            state = 4.0 * k * (H * z["d"] ** 2 + z["Hm"] * z["m"] ** 2)
            cache_tok = 4.0 * k * z["G"] * 2 * z["d"]
            attn_tok = 4.0 * k * H * z["d"]                    # flops per (query, key)
            flops_tok += k * 6.0 * (H * z["d"] ** 2 + z["Hm"] * z["m"] ** 2)
        else:
            state = 4.0 * H * z["dn"] * z["dv"]
            cache_tok = 4.0 * (z["rk"] + z["dr"])
            attn_tok = 2.0 * H * (z["dn"] + z["dr"] + z["dv"])
            flops_tok += 6.0 * H * z["dn"] * z["dv"]
    head = 2.0 * V * W
    if case["call"] == "decode":
        bytes_ = S * (wbytes + head + B * (2 * state + cache_tok * (T + S / 2) + 2 * W)) + 4.0 * B * V
        flops = S * B * (flops_tok + head + attn_tok * (T + S / 2))
    else:
        per = tokens / B
        bytes_ = wbytes + head + B * state + tokens * (cache_tok + 2 * W) + 4.0 * rows * V
        flops = tokens * (flops_tok + attn_tok * per / 2) + rows * head
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # about four times the distance of the path from 64 bits over these ranges: f16 / bf16 operands with f32 sums (1e-3 at most for
    # RWKV, 4e-3 for kemirax; panupel norms read-outs that are nearly zero, which amplifies a rounding: 7e-3 to 3e-2), or f32
    # throughout (2e-5)
    if case["precision"] == 1:
        return {"rel": 1e-4}
    if case["family"].startswith("rwkv"):
        return {"rel": 3e-3}
    return {"rel": 3e-2 if case["family"] == "panupel" else 1.5e-2}


# ----------------------------------------------------------------------------------------------------------------------
# the same models in plain 64-bit torch
# ----------------------------------------------------------------------------------------------------------------------
def _pad(texts, lens, steps):
    n = [a + steps for a in lens]
    T = max(n)
    tok = torch.zeros((len(texts), T), dtype=torch.long, device="cuda")
    for b, t in enumerate(texts):
        tok[b, :n[b]] = torch.from_numpy(t[:n[b]].astype(np.int64)).cuda()
    return tok, torch.tensor(n, device="cuda")


def _layer_norm(x, w, b, eps=1e-5):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, eps)


_NF4 = (-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
        0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0)


def _quantised(w, kind):
    """What a quantised [out, in] matrix multiplies with: blocks of inputs as (min, max) + 8 bits, or absmax + 4-bit levels."""
    n, k = w.shape
    if kind == "Int8":
        b = w.float().reshape(n, -1, 128)
        lo, hi = b.amin(2, keepdim=True), b.amax(2, keepdim=True)
        span = torch.where(hi > lo, hi - lo, torch.ones_like(lo))
        q = torch.floor(((b - lo) / span).clamp(0, 1) * 255.0 + 0.5)
        scale = ((hi - lo) / 255.0).half().double()
        return (q.double() * scale + lo.double()).reshape(n, k)
    b = w.float().reshape(n, -1, 64)
    am = b.abs().amax(2, keepdim=True)
    x = b / torch.where(am > 0, am, torch.ones_like(am))
    lv = torch.tensor(_NF4, dtype=torch.float32, device=w.device)
    q = torch.bucketize(x, (lv[1:] + lv[:-1]) / 2)
    return (lv.half().double()[q] * am.double()).reshape(n, k)


def _rwkv_exact(case, w, tok, n):
    """(residual rows [B, T, C], state [L, N + 2, C] of the first sequence after its last token)."""
    B, T = tok.shape
    C, N = case["width"], HEAD
    H, seven = C // N, case["family"] == "rwkv7"

    def g(name):
        v = w[name]
        if case["quant"] != "none" and name.startswith("blocks.") and name.rsplit(".", 2)[-2] in ("receptance", "key", "value", "gate", "output"):
            return _quantised(v, case["quant"])
        return v.double()

    def vec(name):
        return g(name).reshape(-1)

    def before(h):
        return torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)

    x = _layer_norm(w["emb.weight"][tok].double(), vec("blocks.0.ln0.weight"), vec("blocks.0.ln0.bias"))
    end = int(n[0]) - 1
    states, v_first = [], None
    for l in range(case["layers"]):
        a, f = "blocks.%d.att." % l, "blocks.%d.ffn." % l
        h = _layer_norm(x, vec("blocks.%d.ln1.weight" % l), vec("blocks.%d.ln1.bias" % l))
        d = before(h) - h
        first = h[0, end]
        if seven:
            mix = {c: h + d * vec(a + "x_" + c) for c in "rwkvag"}
            r, k, v = (mix[c] @ g(a + nm + ".weight").T for c, nm in (("r", "receptance"), ("k", "key"), ("v", "value")))
            decay = torch.exp(-0.606531 * torch.sigmoid(vec(a + "w0") + torch.tanh(mix["w"] @ g(a + "w1").T) @ g(a + "w2").T))
            rate = torch.sigmoid(vec(a + "a0") + mix["a"] @ g(a + "a1").T @ g(a + "a2").T)
            gate = torch.sigmoid(mix["g"] @ g(a + "g1").T) @ g(a + "g2").T
            kk = (k * vec(a + "k_k")).view(B, T, H, N)
            kk = kk / kk.norm(dim=-1, keepdim=True).clamp_min(1e-12)
            k = k * (1 + (rate - 1) * vec(a + "k_a"))
            if l == 0:
                v_first = v
            else:
                v = v + (v_first - v) * torch.sigmoid(vec(a + "v0") + mix["v"] @ g(a + "v1").T @ g(a + "v2").T)
            ka = kk * rate.view(B, T, H, N)
        else:
            low = torch.tanh((h + d * vec(a + "time_mix_x")) @ g(a + "time_mix_w1").T).view(B, T, 5, -1)
            low = torch.einsum("btjm,jcm->jbtc", low, g(a + "time_mix_w2"))
            mix = {c: h + d * (vec(a + "time_mix_" + c) + low[j]) for j, c in enumerate("wkvrg")}
            decay = torch.exp(-torch.exp(vec(a + "time_decay") + torch.tanh(mix["w"] @ g(a + "time_decay_w1").T) @ g(a + "time_decay_w2").T))
            r, k, v = (mix[c] @ g(a + nm + ".weight").T for c, nm in (("r", "receptance"), ("k", "key"), ("v", "value")))
            gate = torch.nn.functional.silu(mix["g"] @ g(a + "gate.weight").T)
            u = g(a + "time_first").view(1, H, N, 1)
        del mix
        S = torch.zeros((B, H, N, N), dtype=torch.float64, device="cuda")     # [key, value]; RWKV-7: [value, key]
        out = torch.empty((B, T, C), dtype=torch.float64, device="cuda")
        sh = lambda t, y: y[:, t].reshape(B, H, N)  # noqa: E731
        first_S = None
        for t in range(T):
            if seven:
                sa = -(S * sh(t, kk)[:, :, None, :]).sum(-1)
                S = S * sh(t, decay)[:, :, None, :] + sa[..., None] * sh(t, ka)[:, :, None, :] + sh(t, v)[..., None] * sh(t, k)[:, :, None, :]
                out[:, t] = (S * sh(t, r)[:, :, None, :]).sum(-1).reshape(B, C)
            else:
                kv = sh(t, k)[..., None] * sh(t, v)[:, :, None, :]
                out[:, t] = (sh(t, r)[..., None] * (u * kv + S)).sum(2).reshape(B, C)
                S = kv + sh(t, decay)[..., None] * S
            if t == end:
                first_S = S[0].clone()
        y = out.view(B, T, H, N)
        y = (y - y.mean(-1, keepdim=True)) / torch.sqrt(y.var(-1, unbiased=False, keepdim=True) + 64e-5)
        y = y.reshape(B, T, C) * vec(a + "ln_x.weight") + vec(a + "ln_x.bias")
        if seven:
            bonus = (r * k * vec(a + "r_k")).view(B, T, H, N).sum(-1, keepdim=True)
            y = y + (bonus * v.view(B, T, H, N)).reshape(B, T, C)
        x = x + (y * gate) @ g(a + "output.weight").T
        del out, y, r, k, v, gate, decay
        h = _layer_norm(x, vec("blocks.%d.ln2.weight" % l), vec("blocks.%d.ln2.bias" % l))
        d = before(h) - h
        rows = first_S.transpose(0, 1).reshape(N, C)                          # row i, column (head, j): S[head][i][j]
        states.append(torch.cat([first[None], rows, h[0, end][None]]))
        hid = torch.relu((h + d * vec(f + ("x_k" if seven else "time_mix_k"))) @ g(f + "key.weight").T) ** 2
        y = hid @ g(f + "value.weight").T
        if not seven:
            y = y * torch.sigmoid((h + d * vec(f + "time_mix_r")) @ g(f + "receptance.weight").T)
        x = x + y
    return _layer_norm(x, vec("ln_out.weight"), vec("ln_out.bias")), torch.stack(states)


def _unit(x, eps=_EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, freq, mag=1.0):
    """Half-split rotation of the first 2 len(freq) entries of x [T, heads, dim] by position * freq."""
    k = len(freq)
    ang = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * freq
    c, s = (torch.cos(ang) * mag)[:, None], (torch.sin(ang) * mag)[:, None]
    return torch.cat([x[..., :k] * c - x[..., k:2 * k] * s, x[..., k:2 * k] * c + x[..., :k] * s, x[..., 2 * k:]], -1)


def _panupel_freq():
    f = 5e5 ** (-2.0 * torch.arange(64, dtype=torch.float64, device="cuda") / 128)
    s = _PN_ROT["scaling"]
    keep = ((s["original"] * f / (2 * math.pi) - s["low"]) / (s["high"] - s["low"])).clamp(0, 1)
    return (1 - keep) * f / s["factor"] + keep * f


def _causal(T):
    return torch.ones((T, T), dtype=torch.bool, device="cuda").tril()


def _panupel_exact(case, w, tok, n):
    z = _dims(case)
    B, T = tok.shape
    H, G, d, Hm, m = z["H"], z["G"], z["d"], z["Hm"], z["m"]
    g = lambda name: w[name].double()  # noqa: E731
    x0 = w["embed"][tok].double()
    x = x0
    mask = _causal(T)
    for i, kind in enumerate(_panupel_kinds(case)):
        p = "l%d." % i
        if case["layers"] == 4 and i == 1:
            x = torch.cat([x, x0], -1) @ g("loop.in").T
        h = _unit(x) * g(p + "norm1")
        if kind == "delta":
            q = p + "mix."
            u = {}
            for c in "qkv":
                y, taps = h @ g(q + c).T, g(q + c + ".conv")
                pad = torch.nn.functional.pad(y, (0, 0, z["conv"] - 1, 0))
                u[c] = torch.nn.functional.silu(sum(taps[:, j] * pad[:, j:j + T] for j in range(z["conv"])))
            unit = lambda y: y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
            qq = unit(u["q"].view(B, T, G, d)).repeat_interleave(H // G, 2) * d ** -0.5
            kk = unit(u["k"].view(B, T, G, d)).repeat_interleave(H // G, 2)
            vv = u["v"].view(B, T, H, d)
            beta = torch.sigmoid(h @ g(q + "b").T)
            dec = torch.exp(-torch.exp(g(q + "A_log")) * torch.nn.functional.softplus(h @ g(q + "a").T + g(q + "dt_bias"), threshold=700.0))
            S = torch.zeros((B, H, d, d), dtype=torch.float64, device="cuda")
            out = torch.empty((B, T, H, d), dtype=torch.float64, device="cuda")
            for t in range(T):
                S = S * dec[:, t, :, None, None]
                left = beta[:, t, :, None] * (vv[:, t] - torch.einsum("bhkv,bhk->bhv", S, kk[:, t]))
                S = S + kk[:, t][..., None] * left[:, :, None, :]
                out[:, t] = torch.einsum("bhkv,bhk->bhv", S, qq[:, t])
            y = (_unit(out) * g(q + "norm")).reshape(B, T, H * d) * torch.nn.functional.silu(h @ g(q + "g").T)
            y = y @ g(q + "o").T
        else:
            q, freq = p + "mix.left.", _panupel_freq()
            Q = (_unit(h @ g(q + "q").T) * g(q + "q.norm")).view(B, T, H, d)
            K = (_unit(h @ g(q + "k").T) * g(q + "k.norm")).view(B, T, G, d)
            V = (h @ g(q + "v").T).view(B, T, G, d)
            gate = torch.sigmoid(h @ g(q + "g").T)
            heads = torch.empty((B, T, H, d), dtype=torch.float64, device="cuda")
            for b in range(B):
                Kb, Vb = _turn(K[b], freq).repeat_interleave(H // G, 1), V[b].repeat_interleave(H // G, 1)
                s = torch.einsum("thd,shd->hts", _turn(Q[b], freq), Kb) * d ** -0.5
                s = s.masked_fill(~mask, -math.inf)
                s = torch.cat([s, g(q + "sink")[:, None, None].expand(H, T, 1)], -1).softmax(-1)[..., :-1]
                heads[b] = torch.einsum("hts,shd->thd", s, Vb)
            y = _PN_LEFT * ((heads * gate[..., None]).reshape(B, T, H * d) @ g(q + "o").T)
            q = p + "mix.right."
            qq, kk, vv = ((h @ g(q + c).T).view(B, T, Hm, m) for c in "qkv")
            il = z["cap"] * torch.tanh((h @ g(q + "i").T + g(q + "i.b")) / z["cap"])
            fl = torch.nn.functional.logsigmoid(z["cap"] * torch.tanh((h @ g(q + "f").T + g(q + "f.b")) / z["cap"]))
            S = torch.zeros((B, Hm, m, m), dtype=torch.float64, device="cuda")
            nn, mm = torch.zeros((B, Hm, m), dtype=torch.float64, device="cuda"), torch.zeros((B, Hm), dtype=torch.float64, device="cuda")
            out = torch.empty((B, T, Hm, m), dtype=torch.float64, device="cuda")
            for t in range(T):
                new = torch.maximum(fl[:, t] + mm, il[:, t])
                keep, add = torch.exp(fl[:, t] + mm - new), torch.exp(il[:, t] - new)
                S = keep[..., None, None] * S + (add[..., None] * kk[:, t])[..., None] * vv[:, t][:, :, None, :]
                nn = keep[..., None] * nn + add[..., None] * kk[:, t]
                mm = new
                qt = qq[:, t] * m ** -0.5
                out[:, t] = torch.einsum("bhkv,bhk->bhv", S, qt) / (torch.maximum((nn * qt).sum(-1).abs(), torch.exp(-mm)) + 1e-6)[..., None]
            y = y + _PN_RIGHT * ((_unit(out).reshape(B, T, Hm * m) * g(q + "norm") * torch.sigmoid(h @ g(q + "g").T)) @ g(q + "o").T)
        x = x + z["r"] * _unit(y) * g(p + "norm1b")
        h = _unit(x) * g(p + "norm2")
        y = (torch.nn.functional.silu(h @ g(p + "mlp.gate").T) * (h @ g(p + "mlp.up").T)) @ g(p + "mlp.down").T
        x = x + z["r"] * _unit(y) * g(p + "norm2b")
    return _unit(x) * g("final.norm")


def _kemirax_freq():
    s, base, dims = _KX_ROT["scaling"], _KX_ROT["base"], _KX_ROT["dims"]
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    f = base ** (-2.0 * i / dims)
    turn = lambda t: dims * math.log(s["original"] / (2 * math.pi * t)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(turn(s["fast"])), 0), min(math.ceil(turn(s["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _kemirax_exact(case, w, tok, n):
    z = _dims(case)
    B, T = tok.shape
    H, dn, dr, dv, rk = z["H"], z["dn"], z["dr"], z["dv"], z["rk"]
    g = lambda name: w[name].double()  # noqa: E731
    x = w["embed"][tok].double()
    mask = _causal(T)
    freq, mag = _kemirax_freq()

    def expert(p, h, limit):
        a, u = (h @ g(p + "gate").T).clamp_max(limit), (h @ g(p + "up").T).clamp(-limit, limit)
        return (a * torch.sigmoid(1.702 * a) * (u + 1)) @ g(p + "down").T

    for i in range(2):
        p = "l%d." % i
        h = _unit(x) * g(p + "norm1")
        hs = h + (torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1) - h) * g(p + "shift")
        q = p + "mix."
        if i == 0:
            Q = ((_unit(hs @ g(q + "dq").T) * g(q + "dq.norm")) @ g(q + "uq").T).view(B, T, H, dn + dr)
            kv = hs @ g(q + "dkv").T
            c = _unit(kv[..., :rk]) * g(q + "dkv.norm")
            y = torch.empty((B, T, H, dv), dtype=torch.float64, device="cuda")
            for b in range(B):
                K, V = (c[b] @ g(q + "uk").T).view(T, H, dn), (c[b] @ g(q + "uv").T).view(T, H, dv)
                kr = _turn(kv[b, :, None, rk:], freq, mag)[:, 0]
                s = torch.einsum("thd,shd->hts", Q[b, ..., :dn], K) + torch.einsum("thd,sd->hts", _turn(Q[b, ..., dn:], freq, mag), kr)
                s = (s * (dn + dr) ** -0.5).masked_fill(~mask, -math.inf).softmax(-1)
                y[b] = torch.einsum("hts,shd->thd", s, V)
            y = y.reshape(B, T, H * dv)
        else:
            qq, kk, vv = ((hs @ g(q + n_).T).view(B, T, H, -1) for n_ in "qkv")
            alpha = (torch.sigmoid(hs @ g(q + "a1").T @ g(q + "a2").T + g(q + "a2.b")) ** (1 / z["tau"])).view(B, T, H, dn)
            S = torch.zeros((B, H, dn, dv), dtype=torch.float64, device="cuda")
            y = torch.empty((B, T, H, dv), dtype=torch.float64, device="cuda")
            for t in range(T):
                S = alpha[:, t][..., None] * S + kk[:, t][..., None] * vv[:, t][:, :, None, :]
                y[:, t] = torch.einsum("bhkv,bhk->bhv", S, qq[:, t]) * dn ** -0.5
            y = (_unit(y) * g(q + "norm")).reshape(B, T, H * dv) * torch.nn.functional.silu(hs @ g(q + "g").T)
        y = (y @ g(q + "o").T) * torch.sigmoid(h @ g(p + "rg1").T + g(p + "rg1.b"))
        if i == 0:
            score = (h @ g(p + "mlp.router").T).softmax(-1)
            chosen = (score + g(p + "mlp.correction")).topk(z["top"], -1).indices
            weight = torch.zeros_like(score).scatter(-1, chosen, score.gather(-1, chosen))
            out = h * weight[..., z["E"]:].sum(-1, keepdim=True)
            for e in range(z["E"]):
                at = weight[..., e].nonzero(as_tuple=True)
                if len(at[0]):
                    out[at] += weight[..., e][at][:, None] * expert(p + "mlp.e%d." % e, h[at], z["lim"])
            out = out + torch.sigmoid(h @ g(p + "mlp.shared.sg").T) * expert(p + "mlp.shared.", h, z["slim"])
            y = y + out * torch.sigmoid(h @ g(p + "rg2").T + g(p + "rg2.b"))
        x = x + y
    return _unit(x) * g("final.norm")


def exact(case, seed):
    _, w = _weights(case, seed)
    texts, lens = _texts(case, seed)
    steps = case["steps"]
    tok, n = _pad(texts, lens, steps)
    state = None
    if case["family"].startswith("rwkv"):
        rows, state = _rwkv_exact(case, w, tok, n)
    else:
        rows = (_panupel_exact if case["family"] == "panupel" else _kemirax_exact)(case, w, tok, n)
    head = w["head.weight" if "head.weight" in w else "head"].double()
    B = len(texts)
    if case["call"] == "decode":
        got = torch.stack([rows[torch.arange(B, device="cuda"), n - steps + i] for i in range(steps)]) @ head.T      # [steps, B, V]
        return {"logits": got[-1], "probs": got.softmax(-1).topk(TOP_K, -1).values}
    if case["call"] == "score":
        return {"logits": torch.cat([rows[b, :int(n[b])] for b in range(B)]) @ head.T}
    out = {"logits": rows[torch.arange(B, device="cuda"), n - 1] @ head.T}
    if state is not None and B > 1:
        out["state"] = state
    return out
