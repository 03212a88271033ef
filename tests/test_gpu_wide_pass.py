"""Passes over more than 64 rows of prompts (many-row GEMM, prompt attention) against the CPU oracle, at the edges of their tiles:
128 rows of a GEMM block, 64 rows and keys of an attention tile, 2048 rows of a pass, the shortest run that the prompt attention takes."""
import numpy as np
import pytest

from test_gpu_model import assert_logits_close, make_hf
from homura_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65, 127, 128, 129, 256, 321])
@pytest.mark.parametrize("name,kv", [("qwen2", "F32"), ("llama", "F32"), ("qwen3", "F32"), ("mha", "F32"), ("qwen2", "BF16"), ("qwen3", "BF16")])
def test_prompts_at_the_edges_of_the_tiles(hm, oracle, name, kv, n):
    cfg, d = make_hf(name, max_position_embeddings=512)
    om = oracle.OracleModel.from_hf_dir(d, max_seq_len=512)
    m = hm.HfModel.load(d)
    m.init_kv_cache(512, kv_dtype=hm.DType[kv])
    exact = kv == "F32"
    ids = synth.prompt_ids(13, n + 100, cfg.vocab_size)
    want = om.forward_all(ids)
    tok, lg = m.prefill(ids[:n], want_logits=True)
    assert m.wide_rows() == n
    assert_logits_close(lg, want[n - 1], scale_tol=exact)
    assert not exact or tok == oracle.argmax(want[n - 1])
    # the next portion starts in the middle of a page, of a block of keys, and of nothing
    got, _, _ = m.step([(0, ids[n:], np.arange(100))], want_logits=True)
    assert m.wide_rows() == 100
    assert_logits_close(got, want[n:], scale_tol=exact)
    om.reset()
    om.prefill(ids)
    for layer in range(cfg.num_hidden_layers if exact else 0):
        (gk, gv), (ok, ov) = m.kv_view(layer), om.kv_view(layer)
        np.testing.assert_allclose(gk[0], ok, atol=5e-5)
        np.testing.assert_allclose(gv[0], ov, atol=5e-5)
    m.close()


@pytest.mark.parametrize("name", ["qwen2", "qwen3"])
# One token, 7 (row by row), 8 and 130 rows (tiles) in one batch; short runs from row 107 on, which is no multiple of eight, over row 128,
# and at the end.  All behind contexts of their own; every row's logits.
@pytest.mark.parametrize("before,rows", [([40, 0, 17, 64, 3], [1, 7, 8, 130, 1]), ([0, 9, 5, 33, 16, 1, 70, 2], [107, 7, 7, 7, 1, 3, 20, 5])])
def test_mixed_runs_of_any_length(hm, oracle, name, before, rows):
    cfg, d = make_hf(name, max_position_embeddings=256)
    m = hm.HfModel.load(d)
    n = len(rows)
    m.init_kv_cache(256, batch=n, pool_tokens=n * 256)
    ids = [synth.prompt_ids(50 + i, b + r + 1, cfg.vocab_size) for i, (b, r) in enumerate(zip(before, rows))]
    want = [oracle.OracleModel.from_hf_dir(d, max_seq_len=256).forward_all(t) for t in ids]
    m.step([(i, ids[i][: before[i]], []) for i in range(n) if before[i]], want_logits=False)
    got, greedy, hidden = m.step([(i, ids[i][before[i] : before[i] + rows[i]], np.arange(rows[i])) for i in range(n)], want_logits=True, want_greedy=True, want_hidden=True)
    assert m.wide_rows() == sum(rows)
    ref = np.concatenate([w[b : b + r] for w, b, r in zip(want, before, rows)])
    assert_logits_close(got, ref)
    assert greedy.tolist() == [oracle.argmax(r) for r in ref]
    assert np.isfinite(hidden).all() and np.abs(hidden[-1]).max() > 0
    lg, _ = m.decode_step([int(t[-1]) for t in ids])
    assert_logits_close(lg, np.stack([w[-1] for w in want]))
    m.close()


@pytest.mark.parametrize("kv", ["F32", "BF16"])
@pytest.mark.parametrize("name", ["qwen2", "qwen3"])
def test_attention_in_several_launches(hm, oracle, monkeypatch, name, kv):
    # room for four blocks of 64 keys of f32 pages: sequences of 3, 3, 6 (more than the room by itself) and 1, each launch over the staged
    # blocks of the one in front; and for as many bytes of bf16 pages
    cfg, d = make_hf(name, max_position_embeddings=512)
    block = cfg.num_key_value_heads * 2 * 3 * 64 * cfg.hd * 2
    monkeypatch.setenv("HM_STAGED_KB", str(4 * block // 1024))
    m = hm.HfModel.load(d)
    m.init_kv_cache(512, batch=4, kv_dtype=hm.DType[kv])
    before, rows = [100, 0, 300, 20], [40, 130, 60, 9]
    ids = [synth.prompt_ids(80 + i, b + r, cfg.vocab_size) for i, (b, r) in enumerate(zip(before, rows))]
    want = [oracle.OracleModel.from_hf_dir(d, max_seq_len=512).forward_all(t) for t in ids]
    for i in range(4):
        if before[i]:
            m.step([(i, ids[i][: before[i]], [])], want_logits=False)
    got, _, _ = m.step([(i, ids[i][before[i] :], np.arange(rows[i])) for i in range(4)], want_logits=True)
    assert m.wide_rows() == sum(rows)
    assert_logits_close(got, np.concatenate([w[b:] for w, b in zip(want, before)]), scale_tol=kv == "F32")
    m.close()


def test_tables_of_very_many_runs(hm, oracle):
    # 600 runs of eight rows: more tiles and blocks than the kept tables hold
    cfg, d = make_hf("qwen2", max_position_embeddings=256)
    om = oracle.OracleModel.from_hf_dir(d, max_seq_len=64)
    m = hm.HfModel.load(d)
    m.init_kv_cache(32, batch=600)
    prompts = [synth.prompt_ids(60 + i, 8, cfg.vocab_size) for i in range(7)]
    want = []
    for t in prompts:
        om.reset()
        want.append(om.forward_all(t)[-1])
    for _ in range(2):  # taken, and again
        m.reset_kv_cache()
        got, _, _ = m.step([(i, prompts[i % 7], [7]) for i in range(600)], want_logits=True)
        assert m.wide_rows() == 4800
        assert_logits_close(got, np.stack([want[i % 7] for i in range(600)]))
    m.close()


def test_prompts_of_several_passes(hm, oracle):
    cfg, d = make_hf("qwen2", max_position_embeddings=4352)
    om = oracle.OracleModel.from_hf_dir(d, max_seq_len=4352)
    m = hm.HfModel.load(d)
    m.init_kv_cache(4352)
    ids = synth.prompt_ids(3, 4200, cfg.vocab_size)
    tok, lg = m.prefill(ids, want_logits=True)
    assert m.wide_rows() == 4200
    tok_o, lg_o = om.prefill(ids)
    assert_logits_close(lg, lg_o)
    assert tok == tok_o and m.kv_cache_len() == 4200
    gk, gv = m.kv_view(cfg.num_hidden_layers - 1)
    ok, ov = om.kv_view(cfg.num_hidden_layers - 1)
    np.testing.assert_allclose(gk[0], ok, atol=5e-5)
    np.testing.assert_allclose(gv[0], ov, atol=5e-5)
    m.close()


@pytest.mark.parametrize("gt,bias,norm", [(synth.GGML_Q8_0, False, False), (synth.GGML_Q4_0, False, False), (synth.GGML_Q8_0, True, False), (synth.GGML_Q4_0, False, True)])
@pytest.mark.parametrize("n", [65, 128, 200])
def test_quantised_prompts(hm, oracle, tmp_path, gt, bias, norm, n):
    # whole prompt in one wide pass, and the same in passes of at most 64 rows: the weights are exact in both
    cfg = synth.tiny_config(tie_word_embeddings=False, qkv_bias=bias, qk_norm=norm, head_dim=128 if norm else None, max_position_embeddings=256)
    path = synth.write_gguf_model(str(tmp_path / "m.gguf"), cfg, 7, gt, norm_jitter=0.1)
    om = oracle.OracleModel.from_gguf(path, max_seq_len=256)
    m = hm.HfModel.load_gguf(path)
    m.init_kv_cache(256)
    ids = synth.prompt_ids(21, n + 1, cfg.vocab_size)
    _, want = om.prefill(ids[:n])
    tok, lg = m.prefill(ids[:n], want_logits=True)
    assert m.wide_rows() == n
    ref = max(1.0, float(np.abs(want).max()))
    assert float(np.abs(lg - want).max()) <= 3e-4 * ref  # the bound of the quantised batches
    after = m.decode_step([int(ids[n])])[0][0]
    m.reset_kv_cache()
    for a in range(0, n, 60):
        _, narrow = m.prefill(ids[a : min(n, a + 60)], want_logits=True)
        assert m.wide_rows() == 0
    assert float(np.abs(lg - narrow).max()) <= 3e-4 * ref
    assert float(np.abs(after - m.decode_step([int(ids[n])])[0][0]).max()) <= 3e-4 * ref
    m.close()


@pytest.mark.parametrize("dt", ["Q8_0", "Q4_0"])
def test_norms_of_quantised_prompts_sum_in_64_bits(hm, dt):
    # The output and down projections are zero, so every layer sees the embedding; the value projection picks elements of the normed row: the
    # cached values are the factor's bits.  (f32 sums of the squares put about a third of the rows off by one in the last place.)
    H, I, V, n, kvd = 256, 128, 512, 200, 128
    cfg = hm.TransformerConfig(H, I, 4, 3, 2, V, 1e-6, 1e4, 256, True, 64)

    def blocks(codes):  # [rows, K] whole numbers, scale 1
        c = codes.reshape(-1, 32)
        d = np.broadcast_to(np.float16(1.0).reshape(1).view(np.uint8), (len(c), 2))
        body = c.astype(np.int8).view(np.uint8) if dt == "Q8_0" else (c[:, :16] + 8 | (c[:, 16:] + 8) << 4).astype(np.uint8)
        return np.concatenate([d, body], 1)

    rng = np.random.default_rng(3)
    embed = synth.f32_to_bf16_rne((rng.standard_normal((V, H)) * np.exp(rng.uniform(-3, 3, (V, 1)))).astype(np.float32))
    one = synth.f32_to_bf16_rne(np.ones(H, np.float32))
    tensors = [("model.embed_tokens.weight", hm.DType.BF16, (V, H), embed), ("model.norm.weight", hm.DType.BF16, (H,), one)]
    shapes = {"self_attn.q_proj": (H, H), "self_attn.k_proj": (kvd, H), "self_attn.v_proj": (kvd, H), "self_attn.o_proj": (H, H), "mlp.gate_proj": (I, H), "mlp.up_proj": (I, H), "mlp.down_proj": (H, I)}
    for i in range(3):
        tensors += [(f"model.layers.{i}.{k}_layernorm.weight", hm.DType.BF16, (H,), one) for k in ("input", "post_attention")]
        for name, shape in shapes.items():
            codes = np.zeros(shape, np.int64)
            if "v_proj" in name:
                codes[np.arange(kvd), 2 * np.arange(kvd)] = 1
            tensors.append((f"model.layers.{i}.{name}.weight", hm.DType[dt], shape, blocks(codes)))
    m = hm.HfModel.from_tensors(cfg, tensors)
    m.init_kv_cache(256)
    ids = synth.prompt_ids(8, n, V)
    m.prefill(ids)
    assert m.wide_rows() == n
    x = synth.bf16_to_f32(embed)[np.asarray(ids)]
    inv = np.float32(1) / np.sqrt(((x.astype(np.float64) ** 2).sum(1) / H).astype(np.float32) + np.float32(1e-6))
    want = (x * inv[:, None])[:, ::2].reshape(n, 2, 64).transpose(1, 0, 2)
    for layer in range(3):
        np.testing.assert_array_equal(m.kv_view(layer)[1][0], want)
    m.close()
