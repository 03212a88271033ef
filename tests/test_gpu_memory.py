"""What an engine holds for speed alone (quantised weights a second time, as bf16 terms) makes room for what its calls need."""
import numpy as np
import pytest

from homura_b200 import synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes(hm):
    return hm.dev_mem_info()[0]


class Others:
    """The rest of the GPU taken by others, all but `left` bytes."""

    def __init__(self, hm, left):
        self.buffer = hm.DeviceBuffer(free_bytes(hm) - left)

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.buffer.free()


def load(hm, H, I, heads, kvh, layers=4, V=512, dtype="Q8_0"):
    """A model of random weights; in Q8_0 its copies take 6 bytes per weight."""
    rng = np.random.default_rng(H)

    def weights(rows, k):
        if dtype == "BF16":
            return synth.f32_to_bf16_rne(rng.standard_normal((rows, k), dtype=np.float32) * np.float32(0.02))
        out = np.empty((rows * k // 32, 34), np.uint8)
        out[:, :2] = np.frombuffer(np.float16(0.0005).tobytes(), np.uint8)
        out[:, 2:] = rng.integers(-60, 61, (len(out), 32), np.int8).view(np.uint8)
        return out

    one, hd = synth.f32_to_bf16_rne(np.ones(H, np.float32)), 64
    tensors = [("model.embed_tokens.weight", hm.DType.BF16, (V, H), synth.f32_to_bf16_rne(rng.standard_normal((V, H), dtype=np.float32))), ("model.norm.weight", hm.DType.BF16, (H,), one)]
    for i in range(layers):
        p = f"model.layers.{i}."
        tensors += [(p + k + "_layernorm.weight", hm.DType.BF16, (H,), one) for k in ("input", "post_attention")]
        for name, n, k in [("self_attn.q_proj", heads * hd, H), ("self_attn.k_proj", kvh * hd, H), ("self_attn.v_proj", kvh * hd, H), ("self_attn.o_proj", H, heads * hd), ("mlp.gate_proj", I, H), ("mlp.up_proj", I, H), ("mlp.down_proj", H, I)]:
            tensors.append((p + name + ".weight", hm.DType[dtype], (n, k), weights(n, k)))
    return hm.HfModel.from_tensors(hm.TransformerConfig(H, I, heads, layers, kvh, V, 1e-6, 1e4, 32768, True, hd), tensors)


def large(hm):  # 61 M weights: 65 MB, copies of 365 MB
    return load(hm, 1024, 4096, 16, 4)


def test_a_cache_takes_the_memory_of_the_copies(hm):
    before = free_bytes(hm)
    m = large(hm)
    assert before - free_bytes(hm) > 400 * MB
    ids = synth.prompt_ids(4, 100, 512)
    m.init_kv_cache(256)
    _, want = m.prefill(ids, want_logits=True)
    assert m.wide_rows() == 100
    with Others(hm, 192 * MB):
        m.init_kv_cache(32768)  # 268 MB
        _, got = m.prefill(ids, want_logits=True)
        assert m.wide_rows() == 0
    assert np.abs(got - want).max() <= 3e-4 * max(1.0, float(np.abs(want).max()))
    m.close()


def test_copies_take_an_eighth_of_the_free_memory_at_most(hm):
    with Others(hm, 2048 * MB):
        before = free_bytes(hm)
        m = large(hm)
        assert before - free_bytes(hm) < 150 * MB
        m.init_kv_cache(256)
        m.prefill(synth.prompt_ids(4, 100, 512))
        assert m.wide_rows() == 0
        m.close()


def test_no_copies_for_sizes_that_have_no_wide_passes(hm):
    before = free_bytes(hm)
    m = load(hm, 576, 1536, 9, 3)  # 14 M weights: copies would take 85 MB
    assert before - free_bytes(hm) < 70 * MB
    m.init_kv_cache(256)
    m.prefill(synth.prompt_ids(4, 100, 512))
    assert m.wide_rows() == 0
    m.close()


def test_a_first_long_prompt_allocates_nothing(hm):
    # an allocation takes longer than a short prompt's wide pass saves
    m = large(hm)
    m.init_kv_cache(300)
    m.prefill(synth.prompt_ids(4, 290, 512))  # kernels are loaded
    for tokens, n in ((400, 65), (1000, 900), (250, 128)):
        m.init_kv_cache(tokens)
        before = free_bytes(hm)
        m.prefill(synth.prompt_ids(5, n, 512))
        assert m.wide_rows() == n
        assert before - free_bytes(hm) < 2 * MB  # (what cudaMalloc hands out at least)
    m.close()


def test_long_prompts_without_memory_for_their_scratch(hm):
    m = load(hm, 1024, 4096, 16, 4, layers=2, dtype="BF16")
    ids = synth.prompt_ids(4, 300, 512)
    with Others(hm, 96 * MB):  # the scratch takes more than that
        m.init_kv_cache(2048)
        _, narrow = m.prefill(ids, want_logits=True)
        assert m.wide_rows() == 0
    m.reset_kv_cache()
    _, wide = m.prefill(ids, want_logits=True)  # there is room now
    assert m.wide_rows() == 300
    assert np.abs(narrow - wide).max() <= 1e-4 * max(1.0, float(np.abs(wide).max()))
    m.close()
