"""The tensor-core GEMM (csrc/kq_gemm.cuh) around its tile sizes: 16, 32, 64 and 128 columns, tiles shared between blocks and whole ones, a q6_K
classifier with every tile width, and prompts around the longest pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [12, 13])
@pytest.mark.parametrize("n_in,n_out,ncols", [(256, 2, c) for c in (16, 33, 129)] + [(2048, 384, c) for c in (16, 17, 32, 33, 48, 63, 65, 112, 128, 129, 200)] +
                         [(2560, 19000, c) for c in (17, 129)])
def test_columns_around_the_tiles(pkg, orc, synth, t, n_in, n_out, ncols):
    """Bound as in test_gpu_gemm.py: 4e-6 of the largest result.  Twice, bit for bit: partial results are added in a fixed order."""
    A = synth.matrix(t, n_in, n_out, seed=n_in + n_out + t)
    X = synth.normal_f32(ncols * n_in, 3 + ncols, 1.0).reshape(ncols, n_in)
    X[-1] *= 1e-30  # the factors of a column reach far down
    X[0, n_in // 2] = 3e4  # one activation that dwarfs the others
    Y = np.full((ncols, n_out), np.nan, np.float32)
    again = Y.copy()
    pkg.matmul_(Y, A, X)
    pkg.matmul_(again, A, X)
    assert np.array_equal(Y, again)
    for c in {0, 1, ncols // 2, ncols - 1}:
        want = orc.matmul_f64(A, X[c])
        assert np.abs(Y[c] - want).max() <= 4e-6 * np.abs(want).max(), c


@pytest.mark.parametrize("n_seq", [3, 33, 70, 130])
def test_q6_k_classifier_of_batches(pkg, orc, synth, n_seq):
    cfg = pkg.ModelConfig(512, 768, 1, 4, 2, 1024, 8, 10000.0, False)
    w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=n_seq)
    model = pkg.LanguageModel(cfg, None, w)
    batch = pkg.BatchRunState(model, n_seq)
    ids = synth.tokens(n_seq, 9, 3, cfg.vocab_size)
    batch.decode_next(ids, np.zeros(n_seq, np.int32), want_logits=True)
    oracle = orc.OracleModel(cfg, w)
    for i in {0, 1, n_seq // 2, n_seq - 1}:
        want = oracle.sample_greedy(ids[i:i + 1], 1, want_logits=True)[1][0]
        assert np.abs(batch.logits[i] - want).max() / float(want.max() - want.min()) < 5e-5, i
    batch.close()
    model.close()


def test_a_sequence_has_the_same_bits_in_any_batch(pkg, synth):
    cfg = pkg.ModelConfig(512, 768, 2, 4, 2, 1024, 8, 10000.0, False)
    model = pkg.LanguageModel(cfg, None, synth.model_weights(cfg, dict(synth.ALL(12), w2=13, output=14), seed=5))
    ids = synth.tokens(3 * 130, 9, 3, cfg.vocab_size).reshape(3, 130)
    logits = {}
    for n_seq in (130, 70, 33, 2):
        batch = pkg.BatchRunState(model, n_seq)
        for i in range(3):
            batch.decode_next(ids[i, :n_seq], np.full(n_seq, i, np.int32), want_logits=i == 2)
        logits[n_seq] = np.array(batch.logits)
        batch.close()
        assert np.array_equal(logits[n_seq], logits[130][:n_seq]), n_seq
    model.close()


@pytest.mark.parametrize("n", [10, 512, 513, 514])
def test_prompts_around_the_longest_pass(pkg, orc, synth, n):
    """A pass holds 512 tokens; up to there the last position is in it.  Generation goes on behind it."""
    cfg = pkg.ModelConfig(256, 512, 1, 4, 2, 512, 520, 10000.0, False)
    w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=77)
    ids = synth.tokens(n, 21, 3, cfg.vocab_size)
    tokens, want = orc.OracleModel(cfg, w).sample_greedy(ids, n + 4, want_logits=True)
    model = pkg.LanguageModel(cfg, None, w)
    st = pkg.RunState(model)
    assert pkg.prefill(st, ids, 0) == int(tokens[n - 1])
    assert np.abs(st.logits - want[n - 1]).max() / float(want[n - 1].max() - want[n - 1].min()) < 5e-5
    got, _ = pkg.generate(model, ids, n + 4)
    assert np.array_equal(got, tokens)
    model.close()


def test_prompt_passes_take_the_room_there_is(pkg, synth):
    """With 100 MB left, a prompt of 400 goes through passes of fewer tokens (512 would take 118 MB), not through 200 decode passes."""
    import ctypes as C
    import torch
    from llama2_jl_b200 import _lib as L
    cfg = pkg.ModelConfig(2048, 8192, 1, 16, 16, 512, 600, 10000.0, False)
    w = synth.model_weights(cfg, synth.ALL(12), seed=6)
    models = [pkg.LanguageModel(cfg, None, w) for _ in range(2)]
    roomy, tight = (pkg.RunState(m) for m in models)
    ids = synth.tokens(400, 22, 3, cfg.vocab_size)
    pkg.prefill(roomy, ids, 0)
    torch.cuda.synchronize()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (100 << 20), dtype=torch.uint8, device="cuda")
    pkg.prefill(tight, ids, 0)
    launches = C.c_int64()
    L.check(L.lib().l2b_session_last_launches(tight.session, C.byref(launches)))
    del filler
    torch.cuda.empty_cache()
    assert 13 < launches.value < 100
    assert np.abs(tight.logits - roomy.logits).max() < 2e-5 * float(roomy.logits.max() - roomy.logits.min())
    for m in models:
        m.close()


@pytest.mark.parametrize("n_in,ncols", [(14336, 148), (14336, 149), (28672, 74), (28672, 75)])
def test_columns_of_long_rows(pkg, orc, synth, n_in, ncols):
    """Where a column's blocks are so few that a warp has more than two super-blocks of it (the second of each pair), its values are read a second time.
    Bound as above."""
    A = synth.matrix(12, n_in, 64, seed=n_in)
    X = synth.normal_f32(ncols * n_in, ncols, 1.0).reshape(ncols, n_in)
    Y = np.full((ncols, 64), np.nan, np.float32)
    pkg.matmul_(Y, A, X)
    for c in range(ncols):
        want = orc.matmul_f64(A, X[c])
        assert np.abs(Y[c] - want).max() <= 4e-6 * np.abs(want).max(), c


@pytest.mark.parametrize("dim,hidden,heads,kv", [(256, 14336, 4, 2), (8448, 256, 66, 2)])
def test_prompt_of_long_rows(pkg, orc, synth, dim, hidden, heads, kv):
    """The same behind the feed-forward's activation and behind the residual update and the norm.  Bound as above."""
    cfg = pkg.ModelConfig(dim, hidden, 1, heads, kv, 512, 160, 10000.0, False)
    w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=hidden)
    w.layers[0].rms_att_weight, w.layers[0].rms_ffn_weight = (1 + synth.normal_f32(dim, i, 0.2) for i in (1, 2))
    ids = synth.tokens(150, 23, 3, cfg.vocab_size)
    tokens, want = orc.OracleModel(cfg, w).sample_greedy(ids, 151, want_logits=True)
    model = pkg.LanguageModel(cfg, None, w)
    st = pkg.RunState(model)
    assert pkg.prefill(st, ids, 0) == int(tokens[149])
    assert np.abs(st.logits - want[149]).max() / float(want[149].max() - want[149].min()) < 5e-5
    pkg.transformer_(int(tokens[149]), 150, cfg, st)
    assert np.abs(st.logits - want[150]).max() / float(want[150].max() - want[150].min()) < 5e-5
    model.close()
