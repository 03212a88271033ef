"""Decode steps over keys and values that the caller appended: the weight of every cached row shows in the logits, and a key that is an
infinity takes its row out instead of making the step not a number.

Logits against the same step in numpy at 64 bits, within 1e-4 of the largest logit as the model tests have it.  The rows are bf16 values, so pages of either type
hold them exactly, and values of 8 make the attention the larger part of the hidden state: without one row the logits move by 1e-3 and more."""
import os
import tempfile

import numpy as np
import pytest

from homura_b200 import synth

pytestmark = pytest.mark.gpu

STACKS = {
    "7x64": dict(num_attention_heads=14, num_key_value_heads=2, head_dim=64),
    "8x64": dict(num_attention_heads=32, num_key_value_heads=4, head_dim=64),
    "2x128": dict(num_attention_heads=16, num_key_value_heads=8, head_dim=128, qkv_bias=False, qk_norm=True),
    "6x128": dict(num_attention_heads=6, num_key_value_heads=1, head_dim=128),
}
_made = {}


def _bf16(x):
    return synth.bf16_to_f32(synth.f32_to_bf16_rne(np.ascontiguousarray(x, np.float32)))


def _stack(name):
    if name not in _made:
        cfg = synth.tiny_config(hidden_size=256, intermediate_size=256, num_hidden_layers=1, vocab_size=512, max_position_embeddings=4352, **STACKS[name])
        d = synth.write_hf_model(tempfile.mkdtemp(), cfg, seed=23, norm_jitter=0.1)
        w = {n: (synth.bf16_to_f32(a) if a.dtype == np.uint16 else a).astype(np.float64).reshape(shape) for n, (_, shape, a) in synth.read_safetensors(os.path.join(d, "model.safetensors")).items()}
        _made[name] = cfg, d, w
    return _made[name]


class Step:
    """One step of a one-layer stack at 64 bits; query, key and value of its token are there before the cached rows are chosen."""

    def __init__(self, cfg, w, token, pos, pages):
        self.cfg, self.w = cfg, w
        self.x = w["model.embed_tokens.weight"][token]
        h = self.norm(self.x, "model.layers.0.input_layernorm")
        q, k, v = (self.linear(h, f"model.layers.0.self_attn.{n}_proj").reshape(-1, cfg.hd) for n in "qkv")
        if cfg.qk_norm:
            q, k = self.norm(q, "model.layers.0.self_attn.q_norm"), self.norm(k, "model.layers.0.self_attn.k_norm")
        half = cfg.hd // 2
        angle = pos * cfg.rope_theta ** (-np.arange(half) / half)
        turn = lambda a: np.concatenate([a[:, :half] * np.cos(angle) - a[:, half:] * np.sin(angle), a[:, half:] * np.cos(angle) + a[:, :half] * np.sin(angle)], 1)
        keep = (lambda a: _bf16(a).astype(np.float64)) if pages == "bf16" else (lambda a: a)
        self.q, self.k, self.v = turn(q), keep(turn(k)), keep(v)

    def norm(self, x, name):
        return x / np.sqrt((x * x).mean(-1, keepdims=True) + self.cfg.rms_norm_eps) * self.w[name + ".weight"]

    def linear(self, x, name):
        return self.w[name + ".weight"] @ x + self.w.get(name + ".bias", 0.0)

    def logits(self, keys, values, without=None):
        cfg, kvh = self.cfg, self.cfg.num_key_value_heads
        keys, values = (np.concatenate([a, b[:, None]], 1) for a, b in ((keys, self.k), (values, self.v)))
        s = np.einsum("hgd,hnd->hgn", self.q.reshape(kvh, -1, cfg.hd), keys) / np.sqrt(cfg.hd)
        if without is not None:
            s[..., without] = -np.inf
        p = np.exp(s - s.max(-1, keepdims=True))
        o = np.einsum("hgn,hnd->hgd", p / p.sum(-1, keepdims=True), values).reshape(-1)
        x = self.x + self.linear(o, "model.layers.0.self_attn.o_proj")
        h = self.norm(x, "model.layers.0.post_attention_layernorm")
        gate = self.linear(h, "model.layers.0.mlp.gate_proj")
        x = x + self.linear(gate / (1 + np.exp(-gate)) * self.linear(h, "model.layers.0.mlp.up_proj"), "model.layers.0.mlp.down_proj")
        return self.w["model.embed_tokens.weight" if cfg.tie_word_embeddings else "lm_head.weight"] @ self.norm(x, "model.norm")


def _rows(cfg, n):
    rng = np.random.default_rng(n)
    return (_bf16(rng.standard_normal((cfg.num_key_value_heads, n, cfg.hd)) * size).astype(np.float64) for size in (1.0, 8.0))


def _run(hm, d, cap, pages, token, keys, values):
    m = hm.HfModel.load_with_dtype(d, hm.DType.BF16)
    m.init_kv_cache(cap, kv_dtype=hm.DType.F32 if pages == "f32" else hm.DType.BF16)
    m.kv_append(0, keys[None], values[None], advance=True)
    got, _ = m.decode_step([token])
    m.close()
    return got[0]


# (stack, capacity, cached rows): the short kernel, the streaming one in clusters, and caches that merge through global scratch
CASES = [("7x64", 200, 170), ("7x64", 600, 575), ("7x64", 1800, 1777), ("8x64", 900, 640), ("8x64", 4352, 2303), ("2x128", 800, 784), ("2x128", 1000, 975), ("2x128", 2000, 1103), ("6x128", 700, 687), ("6x128", 2100, 1600)]


@pytest.mark.parametrize("pages", ["f32", "bf16"])
@pytest.mark.parametrize("stack,cap,n", CASES)
def test_every_cached_row_counts(hm, stack, cap, n, pages):
    cfg, d, w = _stack(stack)
    step = Step(cfg, w, 7, n, pages)
    keys, values = _rows(cfg, n)
    want = step.logits(keys, values)
    limit = 1e-4 * max(1.0, float(np.abs(want).max()))
    for row in (0, 15, 16, n // 2, n - 1):
        assert np.abs(step.logits(keys, values, without=row) - want).max() > 4 * limit
    assert np.abs(_run(hm, d, cap, pages, 7, keys, values) - want).max() <= limit


@pytest.mark.parametrize("pages", ["f32", "bf16"])
@pytest.mark.parametrize("stack,cap,n", CASES)
def test_a_key_that_is_an_infinity_takes_its_row_out(hm, stack, cap, n, pages):
    cfg, d, w = _stack(stack)
    kvh = cfg.num_key_value_heads
    for token in range(cfg.vocab_size):  # one whose query heads agree on the sign of some dimension, for every KV head
        step = Step(cfg, w, token, n, pages)
        signs = np.sign(step.q.reshape(kvh, -1, cfg.hd)).sum(1)
        dims = np.abs(signs).argmax(1)
        if (np.abs(signs[np.arange(kvh), dims]) == cfg.num_attention_heads // kvh).all():
            break
    else:
        pytest.fail("no such token")
    keys, values = _rows(cfg, n)
    for row in (3, n // 2, n - 2):
        keys[np.arange(kvh), row, dims] = -np.inf * signs[np.arange(kvh), dims]
    want = step.logits(keys, values)
    assert np.isfinite(want).all()
    assert np.abs(_run(hm, d, cap, pages, token, keys, values) - want).max() <= 1e-4 * max(1.0, float(np.abs(want).max()))


@pytest.mark.parametrize("stack", sorted(STACKS))
def test_a_larger_cache_is_no_less_accurate(hm, stack):
    """The same rows on bf16 pages in a cache whose steps run the short kernel (two pages per CTA, f32 FMAs) and in one whose steps stream (four; tensor cores):
    medians over 24 tokens of the rms error of 512 logits scatter by a few percent, a bit less of precision doubles them."""
    cfg, d, w = _stack(stack)
    n = 490
    keys, values = _rows(cfg, n)
    want = [Step(cfg, w, token, n, "bf16").logits(keys, values) for token in range(24)]
    errors = []
    for cap in (512, 1000):
        m = hm.HfModel.load_with_dtype(d, hm.DType.BF16)
        m.init_kv_cache(cap, kv_dtype=hm.DType.BF16)
        rms = []
        for token in range(24):
            m.reset_kv_cache()
            m.kv_append(0, keys[None], values[None], advance=True)
            got, _ = m.decode_step([token])
            rms.append(float(np.sqrt(((got[0] - want[token]) ** 2).mean())))
        m.close()
        errors.append(float(np.median(rms)))
    assert errors[1] <= 1.25 * errors[0], errors
