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
    assert_logits_close(lg, want[n - 1], scale_tol=exact)
    assert not exact or tok == oracle.argmax(want[n - 1])
    # the next portion starts in the middle of a page, of a block of keys, and of nothing
    got, _, _ = m.step([(0, ids[n:], np.arange(100))], want_logits=True)
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
    ref = np.concatenate([w[b : b + r] for w, b, r in zip(want, before, rows)])
    assert_logits_close(got, ref)
    assert greedy.tolist() == [oracle.argmax(r) for r in ref]
    assert np.isfinite(hidden).all() and np.abs(hidden[-1]).max() > 0
    lg, _ = m.decode_step([int(t[-1]) for t in ids])
    assert_logits_close(lg, np.stack([w[-1] for w in want]))
    m.close()


def test_prompts_of_several_passes(hm, oracle):
    cfg, d = make_hf("qwen2", max_position_embeddings=4352)
    om = oracle.OracleModel.from_hf_dir(d, max_seq_len=4352)
    m = hm.HfModel.load(d)
    m.init_kv_cache(4352)
    ids = synth.prompt_ids(3, 4200, cfg.vocab_size)
    tok, lg = m.prefill(ids, want_logits=True)
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
    ref = max(1.0, float(np.abs(want).max()))
    assert float(np.abs(lg - want).max()) <= 3e-4 * ref  # the bound of the quantised batches
    after = m.decode_step([int(ids[n])])[0][0]
    m.reset_kv_cache()
    for a in range(0, n, 60):
        _, narrow = m.prefill(ids[a : min(n, a + 60)], want_logits=True)
    assert float(np.abs(lg - narrow).max()) <= 3e-4 * ref
    assert float(np.abs(after - m.decode_step([int(ids[n])])[0][0]).max()) <= 3e-4 * ref
    m.close()
