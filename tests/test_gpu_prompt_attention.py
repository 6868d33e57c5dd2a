"""Attention of prompt passes on the tensor cores (csrc/prompt_attention.cuh) against the CPU oracle, through the C ABI: prompts around the
64-position and 128-row tiles, head sizes around its limits, every number of heads per key / value head."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,heads,kv,neox", [(768, 8, 8, True), (1024, 8, 2, False), (512, 16, 16, False), (1024, 8, 1, False), (768, 6, 1, False), (768, 16, 8, False), (256, 16, 8, False)])
@pytest.mark.parametrize("first,second", [(0, 13), (0, 64), (0, 65), (63, 66), (130, 127)])
def test_prompt_passes_against_oracle(pkg, orc, synth, dim, heads, kv, neox, first, second):
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
