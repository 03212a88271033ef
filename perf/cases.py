"""Workloads of the decode engine as its users run them, for timing and for comparing two builds.

Kinds of cases:

* ``request``     one conversation on a uniform bf16 or GGUF model: prefill, then decode_step token by token, every step's logits
                  returned to the host (what the GenerativeModel trait does).  ``new`` 0 is a prompt that is only scored.
* ``batch``       many conversations of ragged lengths: their prompts as one mixed batch, then steps over all of them; greedy, or
                  sampled on the device with the default sampling settings.
* ``attention``   the paged attention kernel by itself on device memory (a plan runner that calls kernel by kernel).
* ``projection``  the six decode projections of the projection sweep on device memory.
* ``tunitar``     a prompt and a few tokens on the latent-attention design through the mixed-batch call.

K-quant files are not here: their projections round the activations to 8 bits, and a sum in another order turns over codes that turn
over others, so that the logits of two right builds differ by 7 % after 22 layers and cannot be compared.

The weights are one seeded random checkpoint per architecture; the seed of a case makes its tokens and activations.  The tokens fed
are given, so that results of one step do not decide the inputs of the next.
"""
from __future__ import annotations

import ctypes
import math
import zlib

import numpy as np
import torch

import homura_b200 as hm

# hidden, intermediate, heads, layers, kv heads, vocab, head_dim, eps, rope theta, tied, qkv bias, qk norm
MODELS = {
    "qwen2.5-0.5b": (896, 4864, 14, 24, 2, 151936, 64, 1e-6, 1e6, True, True, False),
    "qwen2.5-1.5b": (1536, 8960, 12, 28, 2, 151936, 128, 1e-6, 1e6, True, True, False),
    "qwen3-0.6b": (1024, 3072, 16, 28, 8, 151936, 128, 1e-6, 1e6, True, False, True),
    "tinyllama-1.1b": (2048, 5632, 32, 22, 4, 32000, 64, 1e-5, 1e4, False, False, False),
}
POSITIONS = 8192  # rope table: the longest context of these cases
SHAPES = [(896, 1152), (896, 9728), (4864, 896), (1536, 17920), (8960, 1536), (1024, 151936)]
HEADS = {"qwen3-0.6b": (16, 8, 128), "qwen2.5-0.5b": (14, 2, 64), "qwen2.5-1.5b": (12, 2, 128), "tinyllama-1.1b": (32, 4, 64)}
TUNITAR = {"width": 896, "vocab": 151936, "layers": 24, "heads": 14, "dim": 64, "rank": 256, "ff": 7296, "groups": 7, "eps": 1e-6}


def listed():
    return [
        # the smallest call: a short question, a short answer, one user
        {"name": "short-0.5b", "kind": "request", "model": "qwen2.5-0.5b", "weights": "bf16", "kv": "f32", "prompt": 9, "new": 12},
        # the headline configuration: 128 prompt tokens, decoding at batch 1 with the logits of every token
        {"name": "chat-0.5b", "kind": "request", "model": "qwen2.5-0.5b", "weights": "bf16", "kv": "f32", "prompt": 128, "new": 32},
        # a document in the prompt of the small model (odd length, default cache)
        {"name": "document-0.5b", "kind": "request", "model": "qwen2.5-0.5b", "weights": "bf16", "kv": "f32", "prompt": 1999, "new": 0},
        # many users: 64 conversations of the 1.5 B model, prompts of 60 to 400 tokens, bf16 cache
        {"name": "batch64-1.5b", "kind": "batch", "model": "qwen2.5-1.5b", "weights": "bf16", "kv": "bf16", "sequences": 64, "prompt": 400, "new": 24, "sampled": False},
        # a handful of users with the default sampling settings and the default cache
        {"name": "sampled8-1.5b", "kind": "batch", "model": "qwen2.5-1.5b", "weights": "bf16", "kv": "f32", "sequences": 8, "prompt": 100, "new": 24, "sampled": True},
        # a long document, then an answer far into the context; QK-norm, 128-wide heads
        {"name": "long-0.6b", "kind": "request", "model": "qwen3-0.6b", "weights": "bf16", "kv": "bf16", "prompt": 3500, "new": 16},
        # GGUF files: a Q8_0 chat, a Q4_0 document
        {"name": "chat-q8-1.1b", "kind": "request", "model": "tinyllama-1.1b", "weights": "q8_0", "kv": "f32", "prompt": 256, "new": 32},
        {"name": "document-q4-1.1b", "kind": "request", "model": "tinyllama-1.1b", "weights": "q4_0", "kv": "f32", "prompt": 1021, "new": 8},
        # one kernel at a time: attention of a large batch, and far into long contexts on the default cache
        {"name": "attention-64x4096", "kind": "attention", "heads": "qwen3-0.6b", "kv": "bf16", "sequences": 64, "tokens": 4096},
        {"name": "attention-8x16384", "kind": "attention", "heads": "qwen3-0.6b", "kv": "f32", "sequences": 8, "tokens": 16384},
        # one kernel at a time: the projections of a batch of 64
        {"name": "projections-64", "kind": "projection", "rows": 64},
        # the latent-attention design: a prompt and decoding in mixed batches
        {"name": "tunitar-0.5b", "kind": "tunitar", "kv": "bf16", "prompt": 700, "new": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["request"] * 6 + ["batch"] * 3 + ["attention"] * 2 + ["projection", "tunitar"])
    if kind == "request":
        model, weights = rng.choice([("qwen2.5-0.5b", "bf16"), ("qwen2.5-1.5b", "bf16"), ("qwen3-0.6b", "bf16"), ("tinyllama-1.1b", "q8_0"), ("tinyllama-1.1b", "q4_0")])
        return {"kind": kind, "model": model, "weights": weights, "kv": rng.choice(["f32", "bf16"]), "prompt": _log(rng, 2, 4000 if weights == "bf16" else 1500), "new": rng.choice([0, 4, 16, 33])}
    if kind == "batch":
        return {"kind": kind, "model": rng.choice(["qwen2.5-0.5b", "qwen2.5-1.5b", "qwen3-0.6b"]), "weights": "bf16", "kv": rng.choice(["f32", "bf16"]), "sequences": _log(rng, 2, 64), "prompt": _log(rng, 12, 360), "new": rng.randrange(4, 24), "sampled": rng.random() < 0.4}
    if kind == "attention":
        n = _log(rng, 1, 64)
        return {"kind": kind, "heads": rng.choice(sorted(HEADS)), "kv": rng.choice(["f32", "bf16"]), "sequences": n, "tokens": _log(rng, 40, min(32768, 262144 // n))}
    if kind == "projection":
        return {"kind": kind, "rows": rng.randrange(1, 65)}
    return {"kind": kind, "kv": rng.choice(["f32", "bf16"]), "prompt": _log(rng, 3, 1500), "new": rng.randrange(0, 24)}


# ---- checkpoints ---------------------------------------------------------------------------------


def _gen(name):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()))


def _normal(name, shape, std=0.02):
    return (torch.randn(shape, generator=_gen(name), device="cuda", dtype=torch.float32) * std).to(torch.bfloat16)


def _around_one(name, n):
    return (1.0 + 0.1 * torch.randn(n, generator=_gen(name), device="cuda")).to(torch.bfloat16)


def _bytes(t):
    return t.contiguous().view(torch.uint8)


def _quantised(name, n_out, n_in, fmt):
    """Seeded weights of about N(0, 0.02) in GGUF blocks: (bytes, values in 64 bits)."""
    w = torch.randn(n_out * n_in // 32, 32, generator=_gen(name), device="cuda") * 0.02
    d = (w.abs().amax(1, keepdim=True) / (127 if fmt == "q8_0" else 8)).to(torch.float16)
    q = torch.round(w / d.float().clamp_min(1e-12)).clamp(*((-127, 127) if fmt == "q8_0" else (-8, 7))).to(torch.int16)
    values = (d.double() * q.double()).view(n_out, n_in)
    if fmt == "q8_0":
        codes = _bytes(q.to(torch.int8))
    else:
        u = (q + 8).to(torch.uint8)
        codes = u[:, :16] | (u[:, 16:] << 4)
    return torch.cat([_bytes(d), codes], 1), values


def _specs(model):
    """(name, shape, 'w' | 'norm' | 'bias') with norms before the projections, as checkpoints are handed over."""
    H, I, heads, L, kvh, V, hd, _, _, tied, bias, qk_norm = MODELS[model]
    out = [("model.embed_tokens.weight", (V, H), "w"), ("model.norm.weight", (H,), "norm")]
    for i in range(L):
        p = f"model.layers.{i}."
        out += [(p + "input_layernorm.weight", (H,), "norm"), (p + "post_attention_layernorm.weight", (H,), "norm")]
        if qk_norm:
            out += [(p + "self_attn.q_norm.weight", (hd,), "norm"), (p + "self_attn.k_norm.weight", (hd,), "norm")]
        for n, rows in (("q", heads * hd), ("k", kvh * hd), ("v", kvh * hd)):
            if bias:
                out.append((p + f"self_attn.{n}_proj.bias", (rows,), "bias"))
            out.append((p + f"self_attn.{n}_proj.weight", (rows, H), "w"))
        out += [(p + "self_attn.o_proj.weight", (H, heads * hd), "w"), (p + "mlp.gate_proj.weight", (I, H), "w"), (p + "mlp.up_proj.weight", (I, H), "w"), (p + "mlp.down_proj.weight", (H, I), "w")]
    return out + ([] if tied else [("lm_head.weight", (V, H), "w")])


def _format(name, weights):
    """Block format of a projection (None: bf16)."""
    return None if weights == "bf16" or "embed_tokens" in name else weights


_DTYPE = {"q8_0": hm.DType.Q8_0, "q4_0": hm.DType.Q4_0}


def _tensors(model, weights):
    for name, shape, kind in _specs(model):
        fmt = _format(name, weights) if kind == "w" else None
        if fmt:
            yield name, _DTYPE[fmt], shape, _quantised(name, *shape, fmt)[0].cpu().numpy()
        else:
            t = _around_one(name, shape[0]) if kind == "norm" else _normal(name, shape)
            yield name, hm.DType.BF16, shape, t.view(torch.int16).cpu().numpy()


def _tunitar_layers():
    t = TUNITAR
    mixer = {"heads": t["heads"], "dim": t["dim"], "vdim": t["dim"], "kv_rank": t["rank"], "scale": t["dim"] ** -0.5}
    return [{"type": "latent_attention", "mixer": dict(mixer, kv_from=i - 1) if i % 2 else dict(mixer), "mlp": {"kind": "dense", "ff": t["ff"]}} for i in range(t["layers"])]


def _tunitar_tensor(name):
    t = TUNITAR
    W, V, R, q, ff = t["width"], t["vocab"], t["rank"], t["heads"] * t["dim"], t["ff"]
    last = name.split(".", 1)[1] if name[0] == "l" else name
    shape = {"embed": (V, W), "head": (V, W), "mix.q": (q, W), "mix.dkv": (R, W), "mix.uk": (q, R), "mix.uv": (q, R), "mix.g": (q, W), "mix.o": (W, q), "mlp.up": (ff, W), "mlp.down": (W, ff)}.get(last)
    if shape:
        return _normal("tunitar." + name, shape, 1.0 if last == "embed" else shape[1] ** -0.5)
    if last == "shift":
        return torch.rand(W, generator=_gen("tunitar." + name), device="cuda").to(torch.bfloat16)
    return _around_one("tunitar." + name, R if last == "mix.dkv.norm" else W)


def _tunitar_names():
    out = ["embed"]
    for i in range(TUNITAR["layers"]):
        out += [f"l{i}.{n}" for n in ["norm1", "mix.q"] + ([] if i % 2 else ["mix.dkv", "mix.dkv.norm"]) + ["mix.uk", "mix.uv", "mix.g", "mix.o", "ls1", "shift", "norm2", "mlp.up", "mlp.down", "ls2"]]
    return out + ["final.norm", "head"]


_loaded = {}  # the checkpoint that is resident, as a server keeps it: {(model, weights): HfModel}, one at most


def _model(model, weights, batch, length, kv):
    """The resident model with a cache of this shape."""
    key = (model, weights)
    if key not in _loaded:
        for m in _loaded.values():
            m.close()
        _loaded.clear()
        if model == "tunitar":
            import json

            cfg = {"architecture": "Tunitar", "width": TUNITAR["width"], "vocab": TUNITAR["vocab"], "norm": {"groups": TUNITAR["groups"], "eps": TUNITAR["eps"]}, "layers": _tunitar_layers()}
            tensors = ((n, hm.DType.BF16, tuple(t.shape), t.view(torch.int16).cpu().numpy()) for n, t in ((n, _tunitar_tensor(n)) for n in _tunitar_names()))
            _loaded[key] = hm.HfModel.from_config_json(json.dumps(cfg), tensors)
        else:
            H, I, heads, L, kvh, V, hd, eps, theta, tied, _, _ = MODELS[model]
            cfg = hm.TransformerConfig(H, I, heads, L, kvh, V, eps, theta, POSITIONS, tied, hd)
            _loaded[key] = hm.HfModel.from_tensors(cfg, _tensors(model, weights))
        torch.cuda.empty_cache()
    m = _loaded[key]
    shape = (batch, length, kv)
    if getattr(m, "cache_shape", None) != shape:
        m.init_kv_cache(length, batch, hm.DType.F32 if kv == "f32" else hm.DType.BF16)
        m.cache_shape = shape
    return m


# ---- inputs and passes -------------------------------------------------------------------------------


def _lengths(case):
    """Prompt lengths of a batch: from a seventh of the longest upwards, the same for every seed."""
    top, n = case["prompt"], case["sequences"]
    return [max(1, top - (i * 37 % n) * (top - max(1, top // 7)) // max(1, n - 1)) for i in range(n)]


def _tokens(case, seed):
    rng = np.random.default_rng([seed, 17])
    vocab = TUNITAR["vocab"] if case["kind"] == "tunitar" else MODELS[case["model"]][5]
    if case["kind"] == "batch":
        return [rng.integers(0, vocab, n + case["new"], dtype=np.int64) for n in _lengths(case)]
    return rng.integers(0, vocab, case["prompt"] + case["new"], dtype=np.int64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "request":
        ids = _tokens(case, seed)
        m = _model(case["model"], case["weights"], 1, case["prompt"] + case["new"] + 1, case["kv"])
        return {"case": case, "model": m, "prompt": ids[: case["prompt"]], "fed": [np.array([t], np.uint32) for t in ids[case["prompt"] :]]}
    if kind == "batch":
        ids, lens = _tokens(case, seed), _lengths(case)
        m = _model(case["model"], case["weights"], case["sequences"], case["prompt"] + case["new"] + 1, case["kv"])
        entries = [(i, t[:n].astype(np.uint32), np.array([n - 1], np.int32)) for i, (t, n) in enumerate(zip(ids, lens))]
        fed = [np.array([t[n + k] for t, n in zip(ids, lens)], np.uint32) for k in range(case["new"])]
        rng = np.random.default_rng([seed, 23]).integers(1, 1 << 62, case["sequences"], dtype=np.uint64) | np.uint64(1)
        return {"case": case, "model": m, "entries": entries, "fed": fed, "rng": rng}
    if kind == "tunitar":
        ids = _tokens(case, seed)
        m = _model("tunitar", "bf16", 1, case["prompt"] + case["new"] + 1, case["kv"])
        return {"case": case, "model": m, "prompt": ids[: case["prompt"]].astype(np.uint32), "fed": [np.array([t], np.uint32) for t in ids[case["prompt"] :]]}
    for m in _loaded.values():
        m.close()
    _loaded.clear()
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "attention":
        heads, kvh, hd = HEADS[case["heads"]]
        B, T = case["sequences"], case["tokens"]
        pages = -(-T // 16)
        dt = torch.float32 if case["kv"] == "f32" else torch.bfloat16
        k, v = (torch.empty(B * pages, kvh, 16 * hd, device="cuda", dtype=dt) for _ in range(2))
        for t in (k, v):
            for i in range(0, B * pages, 4096):
                t[i : i + 4096] = torch.randn(t[i : i + 4096].shape, generator=g, device="cuda")
        table = torch.randperm(B * pages, generator=g, device="cuda").to(torch.int32).view(B, pages)
        lens = torch.tensor([T - i * 5 % max(1, T // 8) for i in range(B)], dtype=torch.int32, device="cuda")
        q = torch.randn(B, heads * hd, generator=g, device="cuda")
        return {"case": case, "k": k, "v": v, "table": table, "lens": lens, "q": q, "out": torch.empty_like(q), "lib": hm.load_library()}
    lib, M, parts = hm.load_library(), case["rows"], []
    for K, N in SHAPES:
        w = (torch.randn(K, N, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
        x = torch.randn(M, K, generator=g, device="cuda")
        tall = M > 16
        packed = torch.empty(lib.hm_tc_packed_elems(K, N) if tall else -(-N // 128) * K * 128, dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        rc = (lib.hm_pack_bf16_tc if tall else lib.hm_pack_bf16_slabs)(ctypes.c_void_p(w.data_ptr()), K, N, ctypes.c_void_p(packed.data_ptr()), None)
        if rc:
            raise RuntimeError(lib.hm_last_error_global())
        hm.dev_sync()
        parts.append((K, N, x, packed, torch.empty(M, N, device="cuda")))
    return {"case": case, "parts": parts, "tall": M > 16}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("request", "tunitar"):
        m = state["model"]
        m.reset_kv_cache()
        if kind == "request":
            first, logits = m.prefill(state["prompt"], want_logits=True)
        else:
            rows, ids, _ = m.step([(0, state["prompt"], np.array([case["prompt"] - 1], np.int32))], want_logits=True, want_greedy=True)
            first, logits = int(ids[0]), rows[0]
        out, ids = [logits], [first]
        for t in state["fed"]:
            rows, nxt = m.decode_step(t, want_logits=True)
            out.append(rows[0])
            ids.append(int(nxt[0]))
        return {"logits": out, "ids": np.array(ids, np.int64)}
    if kind == "batch":
        m = state["model"]
        m.reset_kv_cache()
        logits, ids, _ = m.step(state["entries"], want_logits=True, want_greedy=True)
        tokens, last, rng = [ids], None, state["rng"].copy()
        for k, t in enumerate(state["fed"]):
            want = k + 1 == len(state["fed"])
            last, nxt = m.decode_step_sampled(t, hm.SamplingConfig(), rng, want) if case["sampled"] else m.decode_step(t, want_logits=want)
            tokens.append(nxt)
        return {"prompts": logits, "ids": np.stack(tokens).astype(np.int64), "last": last}
    st = torch.cuda.current_stream().cuda_stream
    if kind == "attention":
        heads, kvh, hd = HEADS[case["heads"]]
        p = [ctypes.c_void_p(state[n].data_ptr()) for n in ("q", "k", "v", "table", "lens", "out")]
        rc = state["lib"].hm_attn_decode_paged(p[0], p[1], p[2], int(hm.DType.F32 if case["kv"] == "f32" else hm.DType.BF16), p[3], p[4], case["sequences"], heads, kvh, hd, 16, state["table"].shape[1], p[5], ctypes.c_void_p(st))
        if rc:
            raise RuntimeError(state["lib"].hm_last_error_global())
        return state["out"]
    M = case["rows"]
    for K, N, x, w, y in state["parts"]:
        if state["tall"]:
            hm.gemm_bf16_tc((x.data_ptr(), M), w.data_ptr(), N, K=K, y=y.data_ptr(), stream=st)
        else:
            hm.gemv_bf16((x.data_ptr(), M), w.data_ptr(), hm.LAYOUT_SLAB128, K=K, N=N, y=y.data_ptr(), stream=st)
    return [p[4] for p in state["parts"]]


# ---- what a pass cannot do without ------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "attention":
        heads, kvh, hd = HEADS[case["heads"]]
        B, T = case["sequences"], case["tokens"]
        tokens = sum(T - i * 5 % max(1, T // 8) for i in range(B))
        return {"bytes": 2 * tokens * kvh * hd * (4 if case["kv"] == "f32" else 2) + 8 * B * heads * hd, "flops": 4 * tokens * heads * hd}
    if kind == "projection":
        M = case["rows"]
        return {"bytes": sum(2 * K * N + 4 * M * (K + N) for K, N in SHAPES), "flops": sum(2 * M * K * N for K, N in SHAPES)}
    if kind == "tunitar":
        t = TUNITAR
        q = t["heads"] * t["dim"]
        per = t["layers"] * (3 * q * t["width"] + 2 * q * t["rank"] + t["width"] * t["rank"] / 2 + 2 * t["width"] * t["ff"])
        head, scale, kvrow, att = t["vocab"] * t["width"], 2.0, t["layers"] / 2 * t["rank"] * (4 if case["kv"] == "f32" else 2), 4 * t["layers"] * t["heads"] * t["rank"]
    else:
        H, I, heads, L, kvh, V, hd = MODELS[case["model"]][:7]
        per, head = L * (H * hd * (2 * heads + 2 * kvh) + 3 * H * I), V * H
        scale = {"bf16": 2.0, "q8_0": 34 / 32, "q4_0": 18 / 32}[case["weights"]]
        kvrow, att = L * 2 * kvh * hd * (4 if case["kv"] == "f32" else 2), 4 * L * heads * hd
    lens = _lengths(case) if kind == "batch" else [case["prompt"]]
    new, B = case["new"], len(lens)
    rows, wants = sum(lens) + new * B, B + (new * B)
    context = sum(n * (n + 1) / 2 for n in lens) + sum(sum(n + k + 1 for k in range(new)) for n in lens)
    return {"bytes": (1 + new) * (per + head) * scale + sum(n * kvrow for n in lens) + sum(sum((n + k + 1) * kvrow for k in range(new)) for n in lens), "flops": 2 * per * rows + 2 * head * wants + att * context}


def tolerance(case):
    kind = case["kind"]
    if kind in ("attention", "projection"):
        return {"rel": 1e-5, "max": 1e-4}
    if case["kv"] == "bf16":  # keys and values that round to the other neighbour
        return {"rel": 5e-3, "max": 5e-2, "differ": 0.01}
    return {"rel": 5e-5, "max": 5e-4, "differ": 0.01}


# ---- the same in 64 bits ------------------------------------------------------------------------------------


def _cached(x, kv):
    return x.to(torch.bfloat16).double() if kv == "bf16" else x


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _causal(q, k, v, scale):
    """q, k, v [heads, T, .], rows in slices"""
    T, out = q.shape[1], []
    for a in range(0, T, 512):
        b = min(T, a + 512)
        s = q[:, a:b] @ k[:, :b].transpose(1, 2) * scale
        s.masked_fill_(torch.arange(b, device="cuda")[None, :] > torch.arange(a, b, device="cuda")[:, None], -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, :b])
    return torch.cat(out, 1)


def _uniform64(model, weights, kv, sequences, wanted):
    """Logits at the wanted places of every sequence."""
    H, I, heads, L, kvh, V, hd, eps, theta, tied, bias, qk_norm = MODELS[model]
    shapes = {n: (s, kind) for n, s, kind in _specs(model)}

    def W(name):
        s, kind = shapes[name]
        fmt = _format(name, weights) if kind == "w" else None
        return _quantised(name, *s, fmt)[1] if fmt else (_around_one(name, s[0]) if kind == "norm" else _normal(name, s)).double()

    lens = [len(s) for s in sequences]
    ids = torch.tensor(np.concatenate(sequences), device="cuda")
    embed = _normal("model.embed_tokens.weight", (V, H))
    x = embed[ids].double()
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    angle = pos.double()[:, None] * theta ** (-torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)
    cos, sin = (torch.cat([f(angle), f(angle)], 1).float().double()[:, None, :] for f in (torch.cos, torch.sin))
    turn = lambda t: t * cos + torch.cat([-t[..., hd // 2 :], t[..., : hd // 2]], -1) * sin  # noqa: E731
    for i in range(L):
        p = f"model.layers.{i}."
        h = _rms(x, W(p + "input_layernorm.weight"), eps)
        q, k, v = ((h @ W(p + f"self_attn.{n}_proj.weight").T + (W(p + f"self_attn.{n}_proj.bias") if bias else 0)).view(len(pos), -1, hd) for n in "qkv")
        if qk_norm:
            q, k = _rms(q, W(p + "self_attn.q_norm.weight"), eps), _rms(k, W(p + "self_attn.k_norm.weight"), eps)
        q, k, v = turn(q), _cached(turn(k), kv), _cached(v, kv)
        att, at = torch.empty_like(q), 0
        for n in lens:
            a, b, c = (t[at : at + n].transpose(0, 1) for t in (q, k, v))
            att[at : at + n] = _causal(a, b.repeat_interleave(heads // kvh, 0), c.repeat_interleave(heads // kvh, 0), hd**-0.5).transpose(0, 1)
            at += n
        x = x + att.reshape(len(pos), -1) @ W(p + "self_attn.o_proj.weight").T
        h = _rms(x, W(p + "post_attention_layernorm.weight"), eps)
        x = x + (torch.nn.functional.silu(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)) @ W(p + "mlp.down_proj.weight").T
    rows, at = [], 0
    for n, want in zip(lens, wanted):
        rows += [at + j for j in want]
        at += n
    x = _rms(x[torch.tensor(rows, device="cuda")], W("model.norm.weight"), eps)
    return x @ (embed.double() if tied else W("lm_head.weight")).T


def _tunitar64(kv, ids, wanted):
    t = TUNITAR
    T, heads, dim, eps = len(ids), t["heads"], t["dim"], t["eps"]
    W = lambda n: _tunitar_tensor(n).double()  # noqa: E731

    def norm(x, w):
        return _rms(x.view(len(x), t["groups"], -1), 1.0, eps).reshape(x.shape) * w

    x = _tunitar_tensor("embed")[torch.tensor(ids, device="cuda")].double()
    c = None
    for i in range(t["layers"]):
        p = f"l{i}."
        h = norm(x, W(p + "norm1"))
        prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        h = h + (prev - h) * W(p + "shift")
        if i % 2 == 0:
            c = _cached(_rms(h @ W(p + "mix.dkv").T, W(p + "mix.dkv.norm"), eps), kv)
        q, k, v = ((a @ W(p + n).T).view(T, heads, dim).transpose(0, 1) for a, n in ((h, "mix.q"), (c, "mix.uk"), (c, "mix.uv")))
        att = _causal(q, k, v, dim**-0.5).transpose(0, 1).reshape(T, -1)
        x = x + ((att * torch.sigmoid(h @ W(p + "mix.g").T)) @ W(p + "mix.o").T) * W(p + "ls1")
        h = norm(x, W(p + "norm2"))
        x = x + (torch.relu(h @ W(p + "mlp.up").T).square() @ W(p + "mlp.down").T) * W(p + "ls2")
    return norm(x[torch.tensor(wanted, device="cuda")], W("final.norm")) @ W("head").T


def exact(case, seed):
    kind = case["kind"]
    if kind == "request":
        ids, n = _tokens(case, seed), case["prompt"]
        rows = _uniform64(case["model"], case["weights"], case["kv"], [ids], [range(n - 1, n + case["new"])])
        return {"logits": list(rows), "ids": None}
    if kind == "tunitar":
        ids, n = _tokens(case, seed), case["prompt"]
        return {"logits": list(_tunitar64(case["kv"], ids, list(range(n - 1, n + case["new"])))), "ids": None}
    if kind == "batch":
        ids, lens = _tokens(case, seed), _lengths(case)
        rows = _uniform64(case["model"], case["weights"], case["kv"], ids, [[n - 1, n + case["new"] - 1] for n in lens])
        return {"prompts": rows[0::2], "ids": None, "last": rows[1::2]}
    if kind == "attention":
        s = prepare(case, seed)
        heads, kvh, hd = HEADS[case["heads"]]
        out = torch.empty(case["sequences"], heads, hd, device="cuda", dtype=torch.float64)
        for b in range(case["sequences"]):
            n = int(s["lens"][b])
            pages = s["table"][b].long()
            k = s["k"][pages].view(-1, kvh, hd // 4, 16, 4).permute(1, 0, 3, 2, 4).reshape(kvh, -1, hd)[:, :n].double()
            v = s["v"][pages]
            v = (v.view(-1, kvh, 16, hd).transpose(0, 1) if case["kv"] == "f32" else v.view(-1, kvh, hd // 8, 16, 8).permute(1, 0, 3, 2, 4)).reshape(kvh, -1, hd)[:, :n].double()
            q = s["q"][b].double().view(kvh, heads // kvh, hd)
            out[b] = (torch.softmax(q @ k.transpose(1, 2) * hd**-0.5, -1) @ v).reshape(heads, hd)
        return out.reshape(case["sequences"], heads * hd)
    out, g = [], torch.Generator(device="cuda").manual_seed(seed)
    for K, N in SHAPES:
        w = (torch.randn(K, N, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
        x = torch.randn(case["rows"], K, generator=g, device="cuda")
        out.append(x.double() @ w.double())
    return out
