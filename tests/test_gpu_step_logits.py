"""Steps that hand every row's logits to the host: a graph of their own where the head's launch also gives the greedy tokens.  Steps of
five to eight sequences are where the head's kernel changes; every design, against its oracle."""
import dipisun_cases
import dipisun_oracle
import gebilorn_cases
import gebilorn_oracle
import numpy as np
import pulenex_cases
import pulenex_oracle
import pytest
import tunitar_cases
import tunitar_oracle

from homura_b200 import synth

pytestmark = pytest.mark.gpu

# design -> (cases, oracle, further argument of the synthetic models); tolerances as in the tests of the designs
DESIGNS = {
    "tunitar": (tunitar_cases, tunitar_oracle, lambda n: (), 1e-5),
    "dipisun": (dipisun_cases, dipisun_oracle, lambda n: (dipisun_cases.BUCKETS[n],), 3e-5),
    "gebilorn": (gebilorn_cases, gebilorn_oracle, lambda n: (gebilorn_cases.RANKS[n],), 3e-5),
    "pulenex": (pulenex_cases, pulenex_oracle, lambda n: (pulenex_cases.RANKS[n],), 3e-5),
}


def check_steps(m, ids, rows_of, vocab, tol):
    """ids: per sequence prompt and fed tokens; rows_of: per sequence the wanted logits of all places."""
    B, fed = len(ids), 4
    m.step([(b, ids[b][:-fed], []) for b in range(B)], want_logits=False)
    for k in range(fed):
        lg, nxt = m.decode_step([int(t[len(t) - fed + k]) for t in ids], want_logits=True)
        want = np.stack([r[len(t) - fed + k] for r, t in zip(rows_of, ids)])
        assert np.abs(lg - want).max() <= tol * max(1e-3, float(np.abs(want).max())), k
        np.testing.assert_array_equal(nxt, vocab - 1 - lg[:, ::-1].argmax(1))  # ties: the highest index
        assert [m.kv_cache_len(b) for b in range(B)] == [len(t) - fed + k + 1 for t in ids]
    # the tokens of the last step are what the device goes on with
    a = m.decode_greedy_n(None, 3)
    for b in range(B):
        m.reset_kv_cache(b)
    m.step([(b, ids[b], []) for b in range(B)], want_logits=False)
    np.testing.assert_array_equal(a, m.decode_greedy_n(nxt, 3))


@pytest.mark.parametrize("B", [4, 5, 8, 9])
@pytest.mark.parametrize("design", list(DESIGNS))
def test_designs(hm, tmp_path, design, B):
    cases, orc, more, tol = DESIGNS[design]
    cfg = cases.model("mixed")
    w = getattr(synth, design + "_weights")(cfg, 21, *more("mixed"))
    o = orc.Oracle(cfg, {k: synth.bf16_to_f32(v) for k, v in w.items()})
    m = hm.HfModel.load(getattr(synth, f"write_{design}_model")(str(tmp_path / "m"), cfg, 21, w, *more("mixed")))
    m.init_kv_cache(64, batch=B)
    ids = [[int(t) for t in synth.prompt_ids(70 + b, 9 + b, cfg["vocab"])] for b in range(B)]
    check_steps(m, ids, [o.forward(t) for t in ids], cfg["vocab"], tol)
    m.close()


@pytest.mark.parametrize("B", [4, 5, 8, 9])
@pytest.mark.parametrize("weights", ["bf16", "Q8_0 with a bf16 head"])
def test_uniform_stacks(hm, oracle, tmp_path, weights, B):
    cfg = synth.tiny_config()
    if weights == "bf16":
        path = synth.write_hf_model(str(tmp_path), cfg, seed=11, norm_jitter=0.1)
        m, om, tol = hm.HfModel.load(path), oracle.OracleModel.from_hf_dir(path, max_seq_len=64), 1e-4
    else:
        path = synth.write_gguf_model(str(tmp_path / "m.gguf"), cfg, 11, synth.GGML_Q8_0, quant_lm_head=False, norm_jitter=0.1)
        m, om, tol = hm.HfModel.load_gguf(path), oracle.OracleModel.from_gguf(path, max_seq_len=64), 3e-4
    m.init_kv_cache(64, batch=B)
    ids = [[int(t) for t in synth.prompt_ids(70 + b, 9 + b, cfg.vocab_size)] for b in range(B)]
    rows = []
    for t in ids:
        om.reset()
        rows.append(om.forward_all(t))
    check_steps(m, ids, rows, cfg.vocab_size, tol)
    m.close()
