"""Decode steps over caches of every size that changes how the attention of a step is launched: splits without a page, pages
kept in shared memory, streaming clusters, caches of more than 1024 tokens; logits of every step against the CPU oracle.

Tolerance on f32 pages: that of the model tests, 1e-4 of the largest logit (of one where that is less).  On bf16 pages 2e-2: keys and values that lie between two bf16 values go to the
one or the other with the last bit of an f32 sum, 2^-8 of a value each."""
import tempfile

import numpy as np
import pytest

from homura_b200 import synth

pytestmark = pytest.mark.gpu

STACKS = {
    # seven query heads per KV head of 64, gate/up weights of 17 MB: a step's attention asks for them
    "7x64": dict(hidden_size=896, intermediate_size=4864, num_attention_heads=14, num_key_value_heads=2),
    "6x128": dict(hidden_size=768, intermediate_size=512, num_attention_heads=6, num_key_value_heads=1, head_dim=128),
    "2x128": dict(hidden_size=256, intermediate_size=256, num_attention_heads=16, num_key_value_heads=8, head_dim=128, qkv_bias=False, qk_norm=True),
    "3x128": dict(hidden_size=256, intermediate_size=256, num_attention_heads=24, num_key_value_heads=8, head_dim=128),
    "8x128": dict(hidden_size=256, intermediate_size=256, num_attention_heads=32, num_key_value_heads=4, head_dim=128),
    "8x64": dict(hidden_size=256, intermediate_size=256, num_attention_heads=32, num_key_value_heads=4, head_dim=64),
}
_made = {}


def _stack(name):
    if name not in _made:
        cfg = synth.tiny_config(num_hidden_layers=1, vocab_size=512, max_position_embeddings=4352, **STACKS[name])
        _made[name] = cfg, synth.write_hf_model(tempfile.mkdtemp(), cfg, seed=11, norm_jitter=0.1)
    return _made[name]


# (stack, sequences, capacity, prompt, pages): first and last capacities of a rule, prompts that end next to a page's edge
CASES = [
    ("7x64", 1, 20, 9, "f32"), ("7x64", 1, 33, 15, "bf16"), ("7x64", 3, 40, 14, "f32"), ("7x64", 1, 600, 570, "f32"), ("7x64", 2, 900, 878, "bf16"), ("7x64", 1, 1024, 1000, "f32"),
    ("7x64", 1, 1030, 1008, "f32"), ("7x64", 1, 1800, 1775, "bf16"), ("7x64", 1, 4096, 2040, "f32"), ("7x64", 1, 4100, 1030, "f32"), ("7x64", 4, 1500, 300, "f32"),
    ("6x128", 1, 500, 479, "f32"), ("6x128", 2, 1000, 40, "bf16"), ("6x128", 4, 2100, 700, "f32"), ("6x128", 8, 1040, 50, "f32"),
    ("2x128", 1, 700, 681, "f32"), ("2x128", 1, 1000, 975, "bf16"), ("2x128", 1, 1200, 1180, "f32"), ("2x128", 1, 1300, 630, "f32"), ("2x128", 1, 2000, 1100, "bf16"), ("2x128", 2, 1010, 64, "f32"),
    ("3x128", 2, 300, 281, "bf16"), ("3x128", 4, 500, 300, "bf16"), ("3x128", 8, 120, 101, "bf16"), ("3x128", 2, 700, 60, "bf16"),
    ("8x128", 1, 700, 679, "f32"), ("8x128", 1, 4100, 2050, "f32"), ("8x128", 2, 1200, 1190, "f32"), ("8x128", 1, 2560, 1295, "bf16"), ("8x64", 1, 800, 790, "f32"), ("8x64", 1, 4096, 1500, "bf16"), ("8x64", 4, 900, 880, "f32"),
]


@pytest.mark.parametrize("stack,batch,cap,prompt,pages", CASES)
def test_steps_match_the_oracle_whatever_the_cache(hm, oracle, stack, batch, cap, prompt, pages):
    cfg, d = _stack(stack)
    m = hm.HfModel.load_with_dtype(d, hm.DType.BF16)
    m.init_kv_cache(cap, batch=batch, kv_dtype=hm.DType.F32 if pages == "f32" else hm.DType.BF16)
    oms, cur = [], []
    for b in range(batch):
        om = oracle.OracleModel.from_hf_dir(d, max_seq_len=cap)
        ids = synth.prompt_ids(40 + b, max(1, prompt - 7 * b), cfg.vocab_size)
        tok, _ = om.prefill(ids)
        m.prefill(ids, seq=b)
        oms.append(om)
        cur.append(tok)
    for _ in range(min(20, cap - prompt)):
        got, _ = m.decode_step(cur)
        for b in range(batch):
            want = oms[b].decode_step(cur[b])
            err = float(np.abs(got[b] - want).max())
            assert err <= (1e-4 * max(1.0, float(np.abs(want).max())) if pages == "f32" else 2e-2), (b, err)
            cur[b] = oracle.argmax(want)
    m.close()
