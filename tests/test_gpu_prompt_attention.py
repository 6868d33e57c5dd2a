"""Attention of prompt passes on the tensor cores (csrc/prompt_attention.cuh) against the CPU oracle, through the C ABI: prompts around the
64-position and 128-row tiles, head sizes around its limits, every number of heads per key / value head.  Passes as short as these would take
the split kernel by themselves, so each kernel is asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["tiled", "split"])
def kernel(request, monkeypatch):
    monkeypatch.setenv("L2B_PROMPT_ATTENTION", {"tiled": "1", "split": "2"}[request.param])
    return request.param


def test_the_kernel_that_was_asked_for_runs(pkg, synth, monkeypatch):
    """The two differ in the order of their sums, so their bits differ; a head size that the tiled one does not take leaves no choice."""
    for dim, heads, same in ((1024, 8, False), (512, 64, True)):
        cfg = pkg.ModelConfig(dim, 512, 2, heads, heads, 512, 128, 10000.0, False)
        w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=1)
        logits = []
        for asked in ("1", "2", "1"):
            monkeypatch.setenv("L2B_PROMPT_ATTENTION", asked)
            model = pkg.LanguageModel(cfg, None, w)
            st = pkg.RunState(model)
            pkg.prefill(st, synth.tokens(100, 2, 3, cfg.vocab_size), 0)
            logits.append(np.array(st.logits))
            model.close()
        assert np.array_equal(logits[0], logits[2])
        assert np.array_equal(logits[0], logits[1]) == same


@pytest.mark.parametrize("dim,heads,kv,neox", [(768, 8, 8, True), (1024, 8, 2, False), (512, 16, 16, False), (1024, 8, 1, False), (768, 6, 1, False), (768, 16, 8, False), (256, 16, 8, False)])
@pytest.mark.parametrize("first,second", [(0, 13), (0, 64), (0, 65), (63, 66), (130, 127)])
def test_prompt_passes_against_oracle(pkg, orc, synth, kernel, dim, heads, kv, neox, first, second):
    """`first` positions, then `second` more in one pass (head sizes 96, 128, 32, 128, 128 with six heads per key head, 48, 16): logits of the
    last position and of one decoded behind the pass.  Bound: that of the other prompt tests, 5e-5 of the logits' range."""
    cfg = pkg.ModelConfig(dim, 512, 2, heads, kv, 512, 320, 10000.0, neox)
    w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=dim + heads)
    ids = synth.tokens(first + second + 1, 5 + first, 3, cfg.vocab_size)
    _, want = orc.OracleModel(cfg, w).sample_greedy(ids, len(ids), want_logits=True)
    model = pkg.LanguageModel(cfg, None, w)
    st = pkg.RunState(model)
    if first:
        pkg.prefill(st, ids[:first], 0)
    pkg.prefill(st, ids[first:-1], first)
    for pos in (len(ids) - 2, len(ids) - 1):
        if pos == len(ids) - 1:
            pkg.transformer_(int(ids[-1]), pos, cfg, st)
        assert np.abs(st.logits - want[pos]).max() / float(want[pos].max() - want[pos].min()) < 5e-5, pos
    model.close()


@pytest.mark.parametrize("heads,kv", [(8, 8), (8, 4), (8, 2), (8, 1)])
@pytest.mark.parametrize("n", [10, 19])
def test_few_queries_behind_many_positions(pkg, orc, synth, heads, kv, n):
    """Few queries' positions are shared out among up to eight blocks each (the split kernel, one to eight heads per key head).  Bound as above."""
    cfg = pkg.ModelConfig(512, 256, 1, heads, kv, 512, 320, 10000.0, False)
    w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=heads + kv)
    ids = synth.tokens(261 + n, 7 + n, 3, cfg.vocab_size)
    _, want = orc.OracleModel(cfg, w).sample_greedy(ids, len(ids), want_logits=True)
    model = pkg.LanguageModel(cfg, None, w)
    st = pkg.RunState(model)
    pkg.prefill(st, ids[:261], 0)
    pkg.prefill(st, ids[261:], 261)
    assert np.abs(st.logits - want[-1]).max() / float(want[-1].max() - want[-1].min()) < 5e-5
    model.close()


def test_positions_behind_do_not_matter(pkg, synth, kernel):
    """Two prompts that differ from position 60 on, the second with an id there whose embedding is infinite: the rows before it in the cache have
    the same bits, which position 59, fed once more, shows in its logits."""
    cfg = pkg.ModelConfig(1024, 512, 3, 8, 2, 512, 160, 10000.0, False)
    w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=3)
    emb = w.token_embedding_table
    row = emb.data.size // cfg.vocab_size
    data = np.array(emb.data)
    data[7 * row:7 * row + 2] = np.array([0x7C00], np.uint16).view(np.uint8)  # d of the id's first super-block
    w.token_embedding_table = pkg.QuantMatrix(emb.ggml_type, data, emb.in_dim, emb.out_dim)
    model = pkg.LanguageModel(cfg, None, w)
    ids = synth.tokens(100, 4, 8, cfg.vocab_size)
    logits = []
    for tail in (ids[60:], np.concatenate([[7], ids[60:99][::-1]]).astype(ids.dtype)):
        st = pkg.RunState(model)
        try:
            pkg.prefill(st, np.concatenate([ids[:60], tail]), 0)
        except pkg.L2BError:
            assert tail[0] == 7  # its own logits, and those behind, are not numbers
        pkg.transformer_(int(ids[59]), 59, cfg, st)
        logits.append(np.array(st.logits))
    assert np.isfinite(logits[0]).all()
    assert np.array_equal(logits[0], logits[1])
    model.close()
