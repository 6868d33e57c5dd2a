"""GPU parity of the whole per-token path (transformer! and the loop of sample) against the CPU oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")
LOGIT_TOL = 2e-3  # max-abs logit error relative to the logit range (the benchmark's stated tolerance)


def logit_err(got, want):
    return float(np.abs(got - want).max() / (want.max() - want.min()))


def teacher_forced(pkg, model, tokens, n):
    state = pkg.RunState(model)
    out = []
    for pos in range(n):
        pkg.transformer_(int(tokens[pos]), pos, model.config, state)
        out.append(state.logits.copy())
    return np.stack(out)


def test_tiny_f32_golden(pkg, synth):
    """The CPU-runnable configuration: llama2.c-format f32 model, 16 prompt ids + 240 greedy tokens."""
    g = np.load(os.path.join(GOLDEN, "tiny_f32_golden.npz"))
    spec = synth.TINY_F32
    cfg = spec["config"]
    w = synth.model_weights(cfg, spec["types"], seed=int(g["seed"]), tied_output=True)
    model = pkg.LanguageModel(cfg, None, w)
    got, _ = pkg.generate(model, g["prompt"], 256)
    assert np.array_equal(got, g["tokens"]), "greedy token stream differs from the golden stream"
    fed = np.concatenate([g["prompt"][:1], g["tokens"]])
    logits = teacher_forced(pkg, model, fed, 256)
    for p, want in zip(g["positions"], g["logits"]):
        assert logit_err(logits[p], want) < 1e-4
    model.close()


@pytest.mark.parametrize("planes", [3, 2, 1])
def test_reduced_8b_golden(pkg, synth, planes):
    g = np.load(os.path.join(GOLDEN, "reduced_8b_golden.npz"))
    spec = synth.scaled(synth.LLAMA3_8B_Q4_K_S, n_layers=2, vocab_size=4096, seq_len=128)
    cfg = spec["config"]
    w = synth.model_weights(cfg, spec["types"], seed=int(g["seed"]))
    model = pkg.LanguageModel(cfg, None, w, act_planes=planes)
    fed = np.concatenate([g["prompt"][:1], g["tokens"]])
    logits = teacher_forced(pkg, model, fed, 96)
    errs = [logit_err(logits[p], want) for p, want in zip(g["positions"], g["logits"])]
    if planes == 3:
        assert max(errs) < 2e-5, errs
        got, _ = pkg.generate(model, g["prompt"], 96)
        assert np.array_equal(got, g["tokens"])
    elif planes == 2:
        assert max(errs) < LOGIT_TOL / 4, errs
    else:  # single q8_K plane: within the logit tolerance; the free-running stream is not required to match
        assert max(errs) < 5 * LOGIT_TOL, errs
    model.close()


CASES = {
    # name: (spec, layers, vocab, seq_len, n_prompt, n_positions)
    "llama3_gqa4_interleaved": ("LLAMA3_8B_Q4_K_S", 3, 8192, 96, 8, 64),
    "phi3_mha_neox_q5": ("PHI3_MINI_Q5_K_M", 2, 4096, 160, 8, 130),
    "llama70b_gqa8_q4": ("LLAMA2_70B_Q4_K", 1, 2048, 64, 4, 40),
}


@pytest.mark.parametrize("case", list(CASES))
def test_shapes_against_oracle(pkg, orc, synth, case):
    name, layers, vocab, seq, n_prompt, n_pos = CASES[case]
    spec = synth.scaled(getattr(synth, name), n_layers=layers, vocab_size=vocab, seq_len=seq)
    cfg = spec["config"]
    w = synth.model_weights(cfg, spec["types"], seed=100 + layers)
    prompt = synth.tokens(n_prompt, 5, 3, vocab)
    oracle = orc.OracleModel(cfg, w)
    want_tokens, want_logits = oracle.sample_greedy(prompt, n_pos, want_logits=True)
    model = pkg.LanguageModel(cfg, None, w)
    got, _ = pkg.generate(model, prompt, n_pos)
    fed = np.concatenate([prompt[:1], want_tokens])
    logits = teacher_forced(pkg, model, fed, n_pos)
    errs = [logit_err(logits[p], want_logits[p]) for p in range(n_pos)]
    assert max(errs) < 5e-5, max(errs)
    # argmax agrees wherever the oracle's top-1 margin exceeds the measured error
    for p in range(n_pos):
        s = np.sort(want_logits[p])
        if s[-1] - s[-2] > 2 * np.abs(logits[p] - want_logits[p]).max():
            assert int(np.argmax(logits[p])) == int(np.argmax(want_logits[p]))
    assert np.array_equal(got, want_tokens), "greedy stream differs"
    model.close()


@pytest.mark.parametrize("dim,hidden,heads,kv,neox", [(512, 768, 8, 4, False), (768, 1528, 12, 12, True), (1024, 1536, 16, 2, False), (1536, 1544, 12, 12, False), (392, 776, 7, 7, False)])
def test_f32_models_of_other_widths(pkg, orc, synth, dim, hidden, heads, kv, neox):
    """f32 models whose rows take each of the widths that a warp keeps in registers (up to 384, 768, 1536 values), and longer ones, with every prologue and
    epilogue.  A product's error is at most (4 * 12 + 5) * 2^-24 = 3.2e-6 of the sum of its terms' magnitudes; six of them in a row per layer."""
    cfg = pkg.ModelConfig(dim, hidden, 2, heads, kv, 600, 40, 10000.0, neox)
    w = synth.model_weights(cfg, dict(synth.ALL(0), output=0), seed=dim)
    for i, layer in enumerate(w.layers):
        layer.rms_att_weight, layer.rms_ffn_weight = (1 + synth.normal_f32(dim, 10 * i + j, 0.2) for j in (1, 2))
    prompt = synth.tokens(4, 5, 3, cfg.vocab_size)
    want_tokens, want = orc.OracleModel(cfg, w).sample_greedy(prompt, 40, want_logits=True)
    model = pkg.LanguageModel(cfg, None, w)
    got, _ = pkg.generate(model, prompt, 40)
    assert np.array_equal(got, want_tokens)
    logits = teacher_forced(pkg, model, np.concatenate([prompt[:1], want_tokens]), 40)
    assert max(logit_err(logits[p], want[p]) for p in range(40)) < 2e-5
    model.close()


def test_decode_next_session_semantics(pkg, synth):
    """One-step calls, reset, determinism, argument checks."""
    import ctypes as C
    from llama2_jl_b200 import _lib as L
    spec = synth.scaled(synth.LLAMA3_8B_Q4_K_S, n_layers=1, vocab_size=1024, seq_len=32)
    cfg = spec["config"]
    w = synth.model_weights(cfg, spec["types"], seed=3)
    model = pkg.LanguageModel(cfg, None, w)
    prompt = synth.tokens(4, 6, 3, 1024)
    a, _ = pkg.generate(model, prompt, 20)
    b, _ = pkg.generate(model, prompt, 20)
    assert np.array_equal(a, b)
    # the same stream through one-step calls
    state = pkg.RunState(model)
    nxt = C.c_int32()
    tok, stream = int(prompt[0]), []
    for pos in range(20):
        L.check(L.lib().l2b_decode_next(state.session, tok, pos, 0.0, 0.0, C.byref(nxt)))
        tok = int(prompt[pos + 1]) if pos + 1 < 4 else nxt.value
        stream.append(tok)
    assert np.array_equal(np.array(stream), a)
    # temperature sampling is a draw from softmax(logits / T): with u -> 0 it returns the first token with mass
    L.check(L.lib().l2b_decode_next(state.session, tok, 20, 1.0, 0.999, C.byref(nxt)))
    assert 0 <= nxt.value < 1024
    sess = state.session
    assert L.lib().l2b_forward(sess, 5000, 0, None) == L.ERR_BAD_ARG
    assert L.lib().l2b_forward(sess, 1, 32, None) == L.ERR_BAD_ARG
    assert L.lib().l2b_decode_next(sess, 1, 0, 1.0, 1.5, C.byref(nxt)) == L.ERR_BAD_ARG
    assert model.kernels_per_token() == 5 * 1 + 3
    assert model.weight_bytes_per_token() > 0
    model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("arch", ["llama", "phi3"])
def test_native_gguf_loader_matches_python_loader(pkg, synth, tmp_path, arch):
    """l2b_model_load_gguf (the library's own parser, map and upload) gives the same greedy stream and logits as the
    model built from the arrays of the Python loader."""
    from test_host_logic import _write_gguf
    neox = arch == "phi3"
    cfg = pkg.ModelConfig(256, 512, 2, 4, 4 if neox else 2, 64, 512, 500000.0, neox)
    types = dict(synth.ALL(13), output=14) if neox else dict(synth.ALL(12), wv=13, w2=13, output=14)
    w = synth.model_weights(cfg, types, seed=8)
    path = str(tmp_path / f"{arch}.gguf")
    _write_gguf(path, arch, cfg, w, synth, fused=neox)
    a = pkg.load_gguf_model(path, seq_len=64)
    b = pkg.load_gguf_model(path, seq_len=64, native=True)
    assert b.weights is None and b.config == a.config
    prompt = synth.tokens(6, 5, 3, cfg.vocab_size)
    ta, _ = pkg.generate(a, prompt, 32)
    tb, _ = pkg.generate(b, prompt, 32)
    assert np.array_equal(ta, tb)
    sa, sb = pkg.RunState(a), pkg.RunState(b)
    pkg.transformer_(7, 0, a.config, sa)
    pkg.transformer_(7, 0, b.config, sb)
    assert np.array_equal(sa.logits.view(np.uint32), sb.logits.view(np.uint32))
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ["gqa4_interleaved", "mha_neox_q6"])
def test_two_position_prompt_passes_match_one_position_passes(pkg, synth, orc, shape):
    """l2b_generate feeds the prompt two positions per pass (weights streamed once for both).  The stream it produces, the
    KV cache it leaves behind and the logits that follow must agree with the one-position path and with the oracle."""
    if shape == "gqa4_interleaved":
        cfg = pkg.ModelConfig(512, 1024, 3, 8, 2, 512, 64, 10000.0, False)
        types = dict(synth.ALL(12), wv=13, w2=13, output=14)
    else:  # NeoX pairs, every head its own kv head, q6_K layer matrices as in *_K_M files
        cfg = pkg.ModelConfig(768, 1536, 2, 8, 8, 512, 64, 10000.0, True)
        types = dict(synth.ALL(13), wv=14, w2=14, output=14)
    w = synth.model_weights(cfg, types, seed=21)
    prompt = synth.tokens(21, 9, 3, cfg.vocab_size)  # odd length: pairs (0,1) .. (18,19), then 20 alone
    n_pos = 40
    os.environ["L2B_PREFILL_PAIRS"] = "0"
    try:
        single = pkg.LanguageModel(cfg, None, w)
        t1, _ = pkg.generate(single, prompt, n_pos)
    finally:
        del os.environ["L2B_PREFILL_PAIRS"]
    paired = pkg.LanguageModel(cfg, None, w)
    t2, _ = pkg.generate(paired, prompt, n_pos)
    assert np.array_equal(t1, t2)
    want = orc.OracleModel(cfg, w).sample_greedy(prompt, n_pos)
    assert np.array_equal(t2, np.asarray(want, dtype=np.int32))
    # logits at the next position, computed on the caches the two paths filled
    import ctypes as C
    from llama2_jl_b200 import _lib as L
    la, lb = np.zeros(cfg.vocab_size, np.float32), np.zeros(cfg.vocab_size, np.float32)
    L.check(L.lib().l2b_forward(single.device_model().session, int(t1[-1]), n_pos, L.ptr(la)))
    L.check(L.lib().l2b_forward(paired.device_model().session, int(t2[-1]), n_pos, L.ptr(lb)))
    rng = float(la.max() - la.min())
    assert np.abs(la - lb).max() / rng < 1e-5
    single.close()
    paired.close()


@pytest.mark.gpu
def test_prefill_then_decode_matches_generate(pkg, synth):
    """l2b_prefill (the prompt phase as one call, two positions per pass) followed by l2b_decode_next calls gives the stream of
    l2b_generate; a prompt fed in two chunks (second chunk at pos0 > 0) gives it too."""
    import ctypes as C
    from llama2_jl_b200 import _lib as L
    cfg = pkg.ModelConfig(512, 1024, 2, 8, 2, 512, 64, 10000.0, False)
    w = synth.model_weights(cfg, dict(synth.ALL(12), wv=13, w2=13, output=14), seed=3)
    m = pkg.LanguageModel(cfg, None, w)
    prompt = synth.tokens(13, 4, 3, cfg.vocab_size)
    want, _ = pkg.generate(m, prompt, 30)
    for chunks in ([13], [6, 7], [1, 12]):
        st = pkg.RunState(m)  # zeroes the cache
        pos, tok = 0, None
        for n in chunks:
            tok = pkg.prefill(st, prompt[pos:pos + n], pos)
            pos += n
        got = list(prompt[1:]) + [tok]
        nxt = C.c_int32()
        while len(got) < 30:
            L.check(L.lib().l2b_decode_next(st.session, int(got[-1]), len(got), 0.0, 0.0, C.byref(nxt)))
            got.append(nxt.value)
        assert got == [int(t) for t in want], chunks
    with pytest.raises(L.L2BError):
        pkg.prefill(pkg.RunState(m), prompt, 60)  # runs past seq_len
    m.close()


@pytest.mark.gpu
def test_sample_text_with_and_without_prefill(pkg, synth):
    """`sample` prints the same text whether the prompt goes through l2b_prefill or position by position (a max_seq_len
    shorter than the prompt forces the latter), and the text is the decoding of l2b_generate's tokens."""
    import io
    from llama2_jl_b200.tokenizer import CharTokenizer, encode
    tk = CharTokenizer.from_text("abcdefghijklmnopqrstuvwxyz .,")
    vocab = len(tk.id_to_token)
    vocab += vocab % 2
    cfg = pkg.ModelConfig(256, 512, 2, 4, 2, vocab, 48, 10000.0, False)
    w = synth.model_weights(cfg, dict(synth.ALL(12), output=14), seed=12)
    if len(tk.id_to_token) < vocab:
        tk.id_to_token.append("~")
        tk.token_to_id["~"] = vocab - 1
    m = pkg.LanguageModel(cfg, tk, w)
    prompt = "the quick brown fox"
    a, b = io.StringIO(), io.StringIO()
    pkg.sample(m, prompt, temperature=0.0, stop_on_special_token=False, out=a)
    ids = [tk.bos_token_id] + encode(prompt, tk)
    toks, _ = pkg.generate(m, ids, cfg.seq_len)
    text = "".join(tk.id_to_token[int(t)] for t in toks)
    assert a.getvalue().split("\n")[0] == text
    # prefill is skipped when the prompt does not fit into max_seq_len: the per-position path must print the same prefix
    pkg.sample(m, prompt, temperature=0.0, stop_on_special_token=False, max_seq_len=10, out=b)
    assert b.getvalue().split("\n")[0] == text[:10]
    m.close()


@pytest.mark.gpu
def test_llama2c_checkpoint_files(pkg, orc, synth, tmp_path):
    """The CPU-runnable configuration THROUGH its file format: the tiny f32 model written as a llama2.c checkpoint, loaded by
    load_karpathy_model (src/load_karpathy.jl:80-98) and run; then the unshared-classifier variant of the format."""
    from llama2_jl_b200 import load_karpathy as lk
    from llama2_jl_b200.tokenizer import BPETokenizer
    g = np.load(os.path.join(GOLDEN, "tiny_f32_golden.npz"))
    spec = synth.TINY_F32
    cfg = spec["config"]
    w = synth.model_weights(cfg, spec["types"], seed=int(g["seed"]), tied_output=True)
    vocab = [b"t%d" % i for i in range(cfg.vocab_size)]
    tok = BPETokenizer(vocab, {t: i for i, t in enumerate(vocab)}, [0.0] * cfg.vocab_size, 1, 2)
    ck, tk = str(tmp_path / "tiny.bin"), str(tmp_path / "tok.bin")
    lk.write_karpathy_checkpoint(ck, cfg, w)
    lk.write_karpathy_tokenizer(tk, tok)
    model = pkg.load_karpathy_model(ck, tk)
    assert model.config == cfg
    got, _ = pkg.generate(model, g["prompt"], 256)
    assert np.array_equal(got, g["tokens"]), "greedy stream of the model loaded from the file differs from the golden stream"
    model.close()
    # unshared classifier, grouped-query heads: against the oracle on the arrays that were written
    cfg2 = pkg.ModelConfig(288, 768, 2, 6, 3, 1024, 64, 10000.0, False)
    w2 = synth.model_weights(cfg2, synth.ALL(0), seed=5, tied_output=False)
    ck2 = str(tmp_path / "untied.bin")
    lk.write_karpathy_checkpoint(ck2, cfg2, w2, untied=True)
    tok2 = BPETokenizer(vocab[:1024], {t: i for i, t in enumerate(vocab[:1024])}, [0.0] * 1024, 1, 2)
    lk.write_karpathy_tokenizer(tk, tok2)
    m2 = pkg.load_karpathy_model(ck2, tk)
    prompt = synth.tokens(6, 3, 3, 1024)
    want = orc.OracleModel(cfg2, w2).sample_greedy(prompt, 48)
    got2, _ = pkg.generate(m2, prompt, 48)
    assert np.array_equal(got2, want)
    m2.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ["llama_gqa4", "phi3_neox_q6_down", "tiny_dims"])
def test_token_kernel_matches_chain_and_oracle(pkg, orc, synth, shape):
    """The whole token as ONE persistent launch (L2B_TOKEN_KERNEL=1) against the kernel chain and the oracle: same greedy stream,
    logits within reassociation noise, the same stream on every run (arrival counters, ring and ticket state carry over)."""
    from llama2_jl_b200 import _lib as L
    if shape == "llama_gqa4":
        cfg = pkg.ModelConfig(1024, 4608, 3, 8, 2, 1024, 96, 500000.0, False)   # hidden > dim: the down projection is cut in two
        types = dict(synth.ALL(12), wv=13, w2=13, output=14)
    elif shape == "phi3_neox_q6_down":
        cfg = pkg.ModelConfig(768, 2048, 2, 8, 8, 512, 64, 10000.0, True)
        types = dict(synth.ALL(13), wv=14, w2=14, output=14)
    else:  # most blocks have no tile at all in most operations
        cfg = pkg.ModelConfig(256, 512, 2, 4, 2, 64, 64, 500000.0, False)
        types = dict(synth.ALL(12), wv=13, w2=13, output=14)
    w = synth.model_weights(cfg, types, seed=17)
    prompt = synth.tokens(5, 9, 3, cfg.vocab_size)
    n_pos = 48
    chain = pkg.LanguageModel(cfg, None, w)
    t_chain, _ = pkg.generate(chain, prompt, n_pos)
    assert chain.kernels_per_token() == 5 * cfg.n_layers + 3
    os.environ["L2B_TOKEN_KERNEL"] = "1"
    try:
        one = pkg.LanguageModel(cfg, None, w)
        assert one.kernels_per_token() == 1
        runs = [pkg.generate(one, prompt, n_pos)[0] for _ in range(4)]
    finally:
        del os.environ["L2B_TOKEN_KERNEL"]
    assert all(np.array_equal(r, runs[0]) for r in runs)
    want_tokens, want_logits = orc.OracleModel(cfg, w).sample_greedy(prompt, n_pos, want_logits=True)
    if shape != "tiny_dims":  # a 64-word vocabulary over random weights has exact ties; the stream test needs margins
        assert np.array_equal(runs[0], want_tokens) and np.array_equal(t_chain, want_tokens)
    fed = np.concatenate([prompt[:1], want_tokens])
    logits = teacher_forced(pkg, one, fed, n_pos)
    assert max(logit_err(logits[p], want_logits[p]) for p in range(n_pos)) < 5e-5
    chain.close()
    one.close()
