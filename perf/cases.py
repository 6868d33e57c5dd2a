"""Workloads of this library as its users run them, for timing and for comparing results.

A case is a dict of plain values.  Kinds:
  generate  the loop of `sample` in one call: prompt ids, then greedy ids (f32 llama2.c models)
  decode    a chat in progress: ids fed one by one through l2b_decode_next behind a prompt that is in the cache already
  prefill   a prompt, or the next turn of a chat, in one call; its last position's logits and next id
  batch     several sequences advanced in lock step (BatchRunState)
  portion   layer-stack models: a portion of a sequence with logits at chosen places (extend)
  trace     layer-stack models: a request replayed id by id: its prompt, then one position at a time, logits of each
  product   one resident k-quant matrix times some activation vectors that are on the device
Where ids are fed one by one they are given and not chosen, so that two correct implementations walk the same sequence.
Weights are random at the scale of trained ones (standard deviation 0.02, gains around 1)."""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "llama2_jl_b200"  # the package's folder has a dot in its name
    if name not in sys.modules:
        d = os.path.join(ROOT, "llama2.jl_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"), submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


Q4, Q5, Q6 = 12, 13, 14  # ggml types
BYTES = {Q4: 144, Q5: 176, Q6: 210}  # of a block of 256 weights
TYPES = {"q4_K": Q4, "q5_K": Q5, "q6_K": Q6}
_SAME = lambda t: dict(wq=t, wk=t, wv=t, wo=t, w1=t, w2=t, w3=t, emb=t)  # noqa: E731
# dim, hidden, layers, heads, kv heads, vocabulary, positions, RoPE base and form, matrix types
LLAMAS = {
    "8b": (4096, 14336, 32, 32, 8, 128256, 512, 500000.0, False, dict(_SAME(Q4), wv=Q5, w2=Q5, out=Q6)),
    "phi3": (3072, 8192, 32, 32, 32, 32064, 4096, 10000.0, True, dict(_SAME(Q5), out=Q6)),
    "70b": (8192, 28672, 80, 64, 8, 32000, 4096, 10000.0, False, dict(_SAME(Q4), out=Q6)),
}
# width, feed-forward, heads, key/value heads, vocabulary
STACKS = {"2k": (2048, 8192, 16, 4, 32768), "4k": (4096, 14336, 32, 8, 32768)}


def listed():
    return [
        # the smallest model: a few microseconds of work per position, so launches and hand-overs are what counts
        dict(name="tiny_generate", kind="generate", dim=288, hidden=768, layers=6, heads=6, vocab=32000, prompt=16, positions=80),
        # single-user chat, greedy, short context
        dict(name="decode_8b", kind="decode", model="8b", layers=32, past=150, steps=16, temperature=0.0),
        # single-user chat over a long document, sampled as `sample` does by default
        dict(name="decode_phi3_long", kind="decode", model="phi3", layers=32, past=2048, steps=16, temperature=0.9),
        # the widest layers (some of them: all 80 would only repeat them)
        dict(name="decode_70b_layers", kind="decode", model="70b", layers=4, past=300, steps=16, temperature=0.0),
        # a first prompt
        dict(name="prefill_8b_128", kind="prefill", model="8b", layers=32, past=0, tokens=128),
        # the next turn of a chat: a few words behind an earlier exchange
        dict(name="prefill_8b_turn", kind="prefill", model="8b", layers=16, past=211, tokens=29),
        # a long document, first token wanted
        dict(name="prefill_phi3_2048", kind="prefill", model="phi3", layers=32, past=0, tokens=2048),
        # a server's slots, each at a place of its own
        dict(name="batch_8b_24", kind="batch", model="8b", layers=16, seqs=24, past=40, steps=4),
        # prompts of the layer-stack models, logits wanted at some places
        dict(name="savozen_prompt_4k", kind="portion", model="savozen", size="4k", layers=8, tokens=1000, wanted=4, compute="bfloat16"),
        dict(name="perezen_prompt_2k", kind="portion", model="perezen", size="2k", layers=8, tokens=1337, wanted=2, compute="bfloat16"),
        # a recorded request replayed
        dict(name="savozen_trace_2k", kind="trace", model="savozen", size="2k", layers=8, tokens=100, steps=32, compute="bfloat16"),
        # matmul! with several columns on a resident matrix (feed-forward of the 8b shape, an odd number of columns)
        dict(name="product_q5k_37", kind="product", type="q5_K", n_in=4096, n_out=14336, cols=37),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["generate", "decode", "decode", "prefill", "prefill", "batch", "portion", "portion", "trace", "product", "product"])
    if kind == "generate":
        heads = rng.choice([4, 6, 8])
        prompt = _log(rng, 1, 60)
        return dict(kind=kind, dim=heads * rng.choice([16, 48, 64]), hidden=8 * rng.randint(24, 160), layers=rng.randint(2, 8), heads=heads, vocab=2 * rng.randint(150, 16000), prompt=prompt,
                    positions=prompt + rng.randint(10, 100))
    if kind == "product":
        n_in, n_out = 256 * _log(rng, 1, 56), 2 * _log(rng, 32, 8192)
        return dict(kind=kind, type=rng.choice(sorted(TYPES)), n_in=n_in, n_out=n_out, cols=_log(rng, 1, 240))
    if kind in ("decode", "prefill"):
        model = rng.choice(["8b", "8b", "phi3", "phi3", "70b"])
        layers, most = (rng.randint(1, 4) if model == "70b" else rng.randint(2, 16)), 480 if model == "8b" else 2500
        if kind == "decode":
            return dict(kind=kind, model=model, layers=layers, past=_log(rng, 1, most), steps=rng.randint(6, 24), temperature=rng.choice([0.0, 0.9]))
        tokens = _log(rng, 2, most)
        return dict(kind=kind, model=model, layers=layers, past=rng.choice([0, rng.randint(0, most - tokens)]), tokens=tokens)
    if kind == "batch":
        model = rng.choice(["8b", "phi3", "savozen", "perezen"])
        c = dict(kind=kind, model=model, layers=rng.randint(2, 6), seqs=_log(rng, 2, 64), past=0 if model == "perezen" else rng.randint(0, 60), steps=rng.randint(3, 8))
        return dict(c, size="2k", compute="bfloat16") if model in DESIGNS else c
    model = rng.choice(sorted(DESIGNS))
    compute = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
    size, layers = ("2k", rng.randint(2, 4)) if compute == "float32" else (rng.choice(sorted(STACKS)), rng.randint(2, 8))
    if kind == "portion":
        return dict(kind=kind, model=model, size=size, layers=layers, tokens=_log(rng, 2, 200 if compute == "float32" else 1900), wanted=rng.choice([1, 2, 4]), compute=compute)
    return dict(kind=kind, model=model, size=size, layers=layers, tokens=_log(rng, 1, 300), steps=rng.randint(8, 40), compute=compute)


# ---- inputs ---------------------------------------------------------------------------------------------------------------
def _gen(seed, *what):
    g = torch.Generator(device="cuda")
    v = int(seed) & 0xFFFFFFFF
    for w in what:
        v = (v * 1000003 + w + 1) % (1 << 61)
    g.manual_seed(v)
    return g


def _ids(seed, n, vocab, *what):
    return torch.randint(3, vocab, (n,), generator=_gen(seed, 77, *what), device="cuda").cpu().numpy().astype(np.int32)


def _blocks(t, rows, n_in, g):
    """Random k-quant blocks [rows, n_in / 256, bytes] whose weights have mean about 0 and standard deviation about 0.02."""
    n = rows * (n_in // 256)
    b = torch.randint(0, 256, (n, BYTES[t]), dtype=torch.uint8, generator=g, device="cuda")
    d = {Q4: 8e-5, Q5: 4e-5, Q6: 1.5e-5}[t] * (0.5 + torch.rand(n, generator=g, device="cuda"))
    if t == Q6:
        b[:, 208:210] = d.half().view(torch.uint8).view(n, 2)
    else:
        m = d * {Q4: 7.5, Q5: 15.5}[t]  # centres the weights of a block on 0
        b[:, 0:4] = torch.stack([d, m], 1).half().view(torch.uint8).view(n, 4)
    return b.view(rows, n_in // 256, BYTES[t])


def _gain(n, g):
    return 1 + 0.1 * torch.randn(n, generator=g, device="cuda")


ROLES = ("wq", "wk", "wv", "wo", "w1", "w2", "w3")


def _shapes(dim, hidden, heads, kv):
    k = dim // heads * kv
    return dict(wq=(dim, dim), wk=(k, dim), wv=(k, dim), wo=(dim, dim), w1=(hidden, dim), w2=(dim, hidden), w3=(hidden, dim))


def _llama_tensors(c, seed):
    """(two layers, used in turn, top) of the case's llama model: matrices as blocks, or f32 for the tiny one, and gains."""
    if c["kind"] == "generate":
        dim, hidden, heads, kv, vocab, types = c["dim"], c["hidden"], c["heads"], c["heads"], c["vocab"], None
    else:
        dim, hidden, _, heads, kv, vocab, _, _, _, types = LLAMAS[c["model"]]

    def mat(role, i, shape):
        g = _gen(seed, 1, i, len(role) * 7 + ord(role[-1]))
        return torch.randn(shape, generator=g, device="cuda") * shape[1] ** -0.5 if types is None else _blocks(types[role], shape[0], shape[1], g)
    layers = [dict({r: mat(r, i, s) for r, s in _shapes(dim, hidden, heads, kv).items()}, att=_gain(dim, _gen(seed, 2, i)), ffn=_gain(dim, _gen(seed, 3, i))) for i in range(2)]
    top = dict(emb=mat("emb", 9, (vocab, dim)), fin=_gain(dim, _gen(seed, 4)))
    top["out"] = top["emb"] if types is None else mat("out", 9, (vocab, dim))
    return layers, top


def _config(c):
    pkg = _package()
    if c["kind"] == "generate":
        return pkg.ModelConfig(c["dim"], c["hidden"], c["layers"], c["heads"], c["heads"], c["vocab"], max(256, c["positions"]), 10000.0, False)
    dim, hidden, _, heads, kv, vocab, seq_len, base, neox, _ = LLAMAS[c["model"]]
    return pkg.ModelConfig(dim, hidden, c["layers"], heads, kv, vocab, seq_len, base, neox)


def _llama(c, seed):
    pkg = _package()
    cfg = _config(c)
    types = None if c["kind"] == "generate" else LLAMAS[c["model"]][9]
    layers, top = _llama_tensors(c, seed)

    def host(role, t):
        a = t.cpu().numpy()
        return a if types is None else pkg.QuantMatrix(types[role], a.reshape(-1), t.shape[1] * 256, t.shape[0])
    ready = [pkg.TransformerLayerWeights(w["att"].cpu().numpy(), w["ffn"].cpu().numpy(), *(host(r, w[r]) for r in ROLES)) for w in layers]
    emb = host("emb", top["emb"])
    weights = pkg.TransformerWeights(emb, [ready[i % 2] for i in range(c["layers"])], top["fin"].cpu().numpy(), emb if types is None else host("out", top["out"]))
    return pkg.LanguageModel(cfg, None, weights)


def _savozen_raw(c):
    width, ff, heads, _, vocab = STACKS[c["size"]]
    mix = dict(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5, rot=dict(base=500000.0, dims=64))
    return dict(architecture="Savozen", embedding=dict(scale=1.0), norm=dict(eps=1e-5), vocab=vocab, width=width, token_side=dict(dim=width // 16),
                layers=[dict(type="latent_attention", mixer=mix, mlp=dict(kind="dense", ff=ff)) for _ in range(c["layers"])])


def _perezen_raw(c):
    """Layers in threes: attention, mLSTM, attention on the keys and values of the first."""
    width, ff, heads, kv, vocab = STACKS[c["size"]]
    att = dict(heads=heads, kv_heads=kv, dim=64, vdim=128, scale=64 ** -0.5, diff=0.4, rot=dict(base=500000.0, dims=64), mask=dict(size=8192))
    rec = dict(heads=heads // 4, dim=256, vdim=512, gate_cap=15.0)
    mlp = dict(kind="dense", ff=ff)
    return dict(architecture="Perezen", norm=dict(eps=1e-5), vocab=vocab, width=width, max_positions=2048, logit_scale=1.0,
                layers=[dict(type="mlstm", mixer=rec, mlp=None) if i % 3 == 1 else dict(type="attention", mixer=dict(att, kv_from=i - 2) if i % 3 == 2 else att, mlp=mlp)
                        for i in range(c["layers"])])


def _stack_tensors(raw, seed):
    """Weights by tensor name; matrices are bf16 (magnitudes around 1/64) and layers of one shape share them."""
    shared = {}

    def mat(key, out, n_in):
        if key not in shared:
            b = torch.randint(-32768, 32768, (out, n_in), dtype=torch.int16, generator=_gen(seed, 5, len(shared)), device="cuda")
            shared[key] = ((b & -32513) | 0x3C00).view(torch.bfloat16)  # sign and mantissa kept, exponent of two octaves
        return shared[key]

    def vec(shape, mean, std):
        shared[len(shared)] = t = mean + std * torch.randn(shape, generator=_gen(seed, 6, len(shared)), device="cuda")
        return t
    D, V = raw["width"], raw["vocab"]
    w = {"embed": mat("embed", V, D), "head": mat("head", V, D)}
    if raw["architecture"] == "Savozen":
        side = raw["token_side"]["dim"]

        def norm(name):
            w[name], w[name + ".b"], w[name + ".alpha"] = vec(D, 1.0, 0.1), vec(D, 0.0, 0.1), torch.tensor(0.5, device="cuda")
        norm("final.norm")
        w["side.embed"] = mat("side.embed", V, side * len(raw["layers"]))
        for i, l in enumerate(raw["layers"]):
            p, m, ff = f"l{i}.", l["mixer"], l["mlp"]["ff"]
            H, d, r, dv, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            norm(p + "norm1")
            norm(p + "norm2")
            for n, out, n_in in (("q", H * (d + r), D), ("dkv", R + r, D), ("uk", H * d, R), ("uv", H * dv, R), ("g", H * dv, D), ("o", D, H * dv)):
                w[p + "mix." + n] = mat(n, out, n_in)
            w[p + "mix.dkv.norm"], w[p + "mix.sink"] = vec(R, 1.0, 0.1), vec(H, 0.0, 1.0)
            w[p + "mlp.gate"], w[p + "mlp.up"], w[p + "mlp.down"] = mat("gate", ff, D), mat("up", ff, D), mat("down", D, ff)
            w[p + "side.gate"], w[p + "side.proj"], w[p + "side.norm"] = mat("sgate", side, D), mat("sproj", D, side), vec(D, 0.5, 0.05)
        return w
    w["pos"], w["final.norm"] = mat("pos", raw["max_positions"], D), vec(D, 1.0, 0.1)
    for i, l in enumerate(raw["layers"]):
        p, m = f"l{i}.", l["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        w[p + "norm1"], w[p + "norm1b"] = vec(D, 1.0, 0.1), vec(D, 0.5, 0.05)
        w[p + "mix.g"], w[p + "mix.o"] = mat(l["type"] + "g", H * dv, D), mat(l["type"] + "o", D, H * dv)
        if l["type"] == "mlstm":
            for n, rows in (("q", H * d), ("k", H * d), ("v", H * dv), ("i", H), ("f", H)):
                w[p + "mix." + n] = mat("m" + n, rows, D)
            w[p + "mix.norm"], w[p + "mix.i.b"], w[p + "mix.f.b"] = vec(H * dv, 1.0, 0.1), vec(H, 0.0, 0.1), torch.linspace(2.0, 8.0, H, device="cuda")
        else:
            G = m["kv_heads"]
            for n, rows in [("q", H * 2 * d)] + ([("k", G * 2 * d), ("v", G * dv)] if m.get("kv_from") is None else []):
                w[p + "mix." + n], w[p + "mix." + n + ".b"] = mat("a" + n, rows, D), vec(rows, 0.0, 0.1)
                if n != "v":
                    w[p + "mix." + n + ".norm"] = vec(d, 1.0, 0.1)
            for n in ("lq1", "lk1", "lq2", "lk2"):
                w[p + "mix." + n] = vec(d, 0.0, 0.1)
        if l["mlp"]:
            ff = l["mlp"]["ff"]
            w[p + "norm2"], w[p + "norm2b"] = vec(D, 1.0, 0.1), vec(D, 0.5, 0.05)
            w[p + "mlp.gate"], w[p + "mlp.up"], w[p + "mlp.down"] = mat("gate", ff, D), mat("up", ff, D), mat("down", D, ff)
    return w


DESIGNS = {"savozen": _savozen_raw, "perezen": _perezen_raw}


def _stack(c, seed):
    pkg = _package()
    raw = DESIGNS[c["model"]](c)
    host, weights = {}, pkg.StackWeights()
    for name, t in _stack_tensors(raw, seed).items():
        if t.data_ptr() not in host:  # shared matrices come to the host once
            host[t.data_ptr()] = t.view(torch.int16).cpu().numpy().view(np.uint16) if t.dtype == torch.bfloat16 else t.cpu().numpy()
        weights[name] = host[t.data_ptr()]
    return pkg.LanguageModel(pkg.StackConfig(raw, 2048, c["compute"]), None, weights)


def _vocab(c):
    return c["vocab"] if "vocab" in c else LLAMAS[c["model"]][5] if c["model"] in LLAMAS else STACKS[c["size"]][4]


def _wanted(c):
    n, k = c["tokens"], min(c["wanted"], c["tokens"])
    return [(i + 1) * n // k - 1 for i in range(k)]


def _batch_script(c, seed):
    """Ids [sequences, past + steps]; sequence i took its slot over `late[i]` steps after the first ones began."""
    ids = _ids(seed, c["seqs"] * (c["past"] + c["steps"]), _vocab(c)).reshape(c["seqs"], -1)
    late = np.random.RandomState(seed & 0x7FFFFFFF).randint(0, c["past"] // 2 + 1, c["seqs"])
    return ids, late


def prepare(case, seed):
    c, pkg = case, _package()
    kind = c["kind"]
    if kind == "product":
        t = TYPES[c["type"]]
        a = _blocks(t, c["n_out"], c["n_in"], _gen(seed, 1)).cpu().numpy()
        x = torch.randn((c["cols"], c["n_in"]), generator=_gen(seed, 2), device="cuda")
        return _Product(pkg, t, a, c, x)
    model = _stack(c, seed) if c.get("model") in DESIGNS else _llama(c, seed)
    if kind == "batch":
        ids, late = _batch_script(c, seed)
        batch = pkg.BatchRunState(model, c["seqs"])
        for i in range(c["past"]):  # a slot that is taken over late holds something else until then
            batch.decode_next(ids[:, i], np.where(i < late, i, i - late))
        return dict(c=c, model=model, batch=batch, ids=ids, late=late)
    ids = _ids(seed, c.get("prompt", 0) + c.get("past", 0) + c.get("tokens", 0) + c.get("steps", 0), _vocab(c))
    state = pkg.RunState(model)
    if c.get("past"):
        pkg.prefill(state, ids[:c["past"]])
    uniforms = np.random.RandomState(seed & 0x7FFFFFFF).random_sample(c.get("steps", 0))
    return dict(c=c, model=model, state=state, ids=ids, uniforms=uniforms)


class _Product:
    """A resident matrix and the vectors it is applied to."""

    def __init__(self, pkg, t, a, c, x):
        from llama2_jl_b200 import _lib as L
        self.c, self.L, self.x, self.handle = c, L, x, C.c_void_p()
        self.y = torch.empty((c["cols"], c["n_out"]), device="cuda")
        L.check(L.lib().l2b_matrix_create(t, L.ptr(a), c["n_in"], c["n_out"], 1, C.byref(self.handle)))

    def run(self):
        L, stream = self.L, torch.cuda.current_stream().cuda_stream
        if self.c["cols"] >= 4 and self.c["type"] != "q6_K":
            L.check(L.lib().l2b_matrix_matmul_device(self.handle, 0, self.x.data_ptr(), self.c["cols"], self.y.data_ptr(), stream))
        else:
            for i in range(self.c["cols"]):
                L.check(L.lib().l2b_matrix_matvec_device(self.handle, 0, self.x[i].data_ptr(), self.y[i].data_ptr(), 0, stream))
        return self.y

    def __del__(self):
        self.L.lib().l2b_matrix_destroy(self.handle)


def run(state):
    if isinstance(state, _Product):
        return state.run()
    pkg, c = _package(), state["c"]
    from llama2_jl_b200 import _lib as L
    kind, ids = c["kind"], state["ids"]
    if kind == "generate":
        tokens, _ = pkg.generate(state["model"], ids, c["positions"])
        logits = state["state"].logits
        L.check(L.lib().l2b_session_logits(state["state"].session, L.ptr(logits)))
        return dict(tokens=tokens, logits=logits)
    if kind == "decode":
        s, nxt, chosen = state["state"], C.c_int32(), []
        for i in range(c["steps"]):
            pos = c["past"] + i
            L.check(L.lib().l2b_decode_next(s.session, int(ids[pos]), pos, c["temperature"], float(state["uniforms"][i]), C.byref(nxt)))
            chosen.append(nxt.value)
        L.check(L.lib().l2b_session_logits(s.session, L.ptr(s.logits)))
        # sampled ids hang on the last bit of a running sum over the vocabulary: the distribution that they come from is compared
        return dict(logits=s.logits) if c["temperature"] else dict(tokens=np.array(chosen), logits=s.logits)
    if kind == "prefill":
        s = state["state"]
        nxt = pkg.prefill(s, ids[c["past"]:], c["past"])
        return dict(next=nxt, logits=s.logits)
    if kind == "batch":
        b, late, chosen = state["batch"], state["late"], []
        for i in range(c["past"], c["past"] + c["steps"]):
            chosen.append(b.decode_next(ids[:, i], i - late, want_logits=i + 1 == c["past"] + c["steps"]))
        return dict(logits=b.logits) if c["model"] in DESIGNS else dict(tokens=np.stack(chosen), logits=b.logits)
    s = state["state"]
    if kind == "portion":
        return dict(logits=pkg.extend(s, ids, 0, _wanted(c)))
    rows = [pkg.extend(s, ids[:c["tokens"]], 0, [c["tokens"] - 1])]
    rows += [pkg.extend(s, ids[i:i + 1], i, [0]) for i in range(c["tokens"], len(ids))]
    return dict(logits=np.concatenate(rows))


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def _dense(c):
    """(weights, their bytes) of the layers and of the classifier."""
    if c["kind"] == "generate":
        n = sum(a * b for a, b in _shapes(c["dim"], c["hidden"], c["heads"], c["heads"]).values()) * c["layers"]
        h = c["vocab"] * c["dim"]
        return n, 4 * n, h, 4 * h
    if c["model"] in LLAMAS:
        dim, hidden, _, heads, kv, vocab, _, _, _, types = LLAMAS[c["model"]]
        s = _shapes(dim, hidden, heads, kv)
        n = c["layers"] * sum(a * b for a, b in s.values())
        return n, c["layers"] * sum(a * b * BYTES[types[r]] // 256 for r, (a, b) in s.items()), vocab * dim, vocab * dim * BYTES[types["out"]] // 256
    raw, n = DESIGNS[c["model"]](c), 0
    D = raw["width"]
    for l in raw["layers"]:
        m = l["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if l["type"] == "latent_attention":
            n += D * (H * (d + m["rot_dim"]) + m["kv_rank"] + m["rot_dim"] + 2 * H * dv) + H * (d + dv) * m["kv_rank"] + 2 * D * raw["token_side"]["dim"]
        elif l["type"] == "mlstm":
            n += D * (H * (2 * d + 2) + 3 * H * dv)
        else:
            n += D * (2 * H * d + 2 * H * dv + (0 if m.get("kv_from") is not None else m["kv_heads"] * (2 * d + dv)))
        n += 3 * D * (l["mlp"]["ff"] if l["mlp"] else 0)
    return n, 2 * n, raw["vocab"] * D, 2 * raw["vocab"] * D


def _mixing(c, pos):
    """(flops, bytes of cache or state) of the mixers of one token at position pos."""
    if c["kind"] == "generate" or c["model"] in LLAMAS:
        dim, heads, kv = (c["dim"], c["heads"], c["heads"]) if c["kind"] == "generate" else (LLAMAS[c["model"]][i] for i in (0, 3, 4))
        return 4 * dim * (pos + 1) * c["layers"], 8 * dim // heads * kv * (pos + 1) * c["layers"]
    flops = size = 0
    wide = 4 if c["compute"] == "float32" else 2
    for l in DESIGNS[c["model"]](c)["layers"]:
        m = l["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if l["type"] == "latent_attention":
            flops += 2 * H * (pos + 1) * (d + m["rot_dim"] + dv)
            size += wide * (pos + 1) * (m["kv_rank"] + m["rot_dim"])
        elif l["type"] == "mlstm":
            flops += 4 * H * d * dv
            size += 8 * H * d * dv
        else:
            flops += 4 * H * (pos + 1) * (d + dv)
            size += wide * (pos + 1) * m["kv_heads"] * (2 * d + dv)
    return flops, size


def work(case):
    c, kind = case, case["kind"]
    if kind == "product":
        n = c["n_in"] * c["n_out"]
        return dict(bytes=n * BYTES[TYPES[c["type"]]] // 256 + 4 * c["cols"] * (c["n_in"] + c["n_out"]), flops=2 * n * c["cols"])
    n, size, h, hsize = _dense(c)
    flops = moved = 0

    def several(first, count, heads_wanted):  # one pass over the weights for all of them
        nonlocal flops, moved
        f = [_mixing(c, p) for p in (first, first + count - 1)]
        flops += 2 * n * count + 2 * h * heads_wanted + count * (f[0][0] + f[1][0]) // 2
        moved += size + hsize + f[1][1] + 4 * heads_wanted * _vocab(c)
    if kind in ("generate", "trace"):
        prompt = c["prompt"] if kind == "generate" else c["tokens"]
        several(0, prompt, 1)
        for p in range(prompt, c["positions"] if kind == "generate" else prompt + c["steps"]):
            several(p, 1, 1)
    elif kind == "decode":
        for p in range(c["past"], c["past"] + c["steps"]):
            several(p, 1, 1)
    elif kind == "prefill":
        several(c["past"], c["tokens"], 1)
    elif kind == "portion":
        several(0, c["tokens"], min(c["wanted"], c["tokens"]))
    else:
        for i in range(c["steps"]):
            f, b = _mixing(c, c["past"] * 3 // 4 + i)
            flops += c["seqs"] * (2 * n + 2 * h + f)
            moved += size + hsize + c["seqs"] * b
        moved += 4 * c["seqs"] * _vocab(c)
    return dict(bytes=moved, flops=flops)


def tolerance(case):
    # About four times what is measured against exact(): 2e-7 for one product in 32 bits, up to 6e-6 through 32 layers of them, up to
    # 1e-2 with bf16 operands.
    c = case
    if c["kind"] == "product":
        return dict(rel=1e-6, max=1e-5)
    if c["kind"] != "generate" and c["model"] in DESIGNS and c["compute"] == "bfloat16":
        return dict(rel=3e-2, max=3e-1)
    return dict(rel=2e-5, max=2e-4, differ=0.01)


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------
def _dequant(t, b):
    """Blocks [rows, blocks, bytes] -> f64 [rows, 256 * blocks]."""
    n = b.shape[0] * b.shape[1]
    b = b.reshape(n, -1)
    half = lambda lo: b[:, lo:lo + 2].contiguous().view(torch.float16).double()  # noqa: E731
    if t == Q6:
        ql, qh = b[:, :128].view(n, 2, 64).short(), b[:, 128:192].view(n, 2, 32).short()
        sc = b[:, 192:208].contiguous().view(torch.int8).double().view(n, 2, 8)
        q = torch.stack([(ql[..., :32] & 15) | ((qh & 3) << 4), (ql[..., 32:] & 15) | ((qh >> 2 & 3) << 4),
                         (ql[..., :32] >> 4) | ((qh >> 4 & 3) << 4), (ql[..., 32:] >> 4) | ((qh >> 6) << 4)], 2) - 32
        w = half(208).view(n, 1, 1, 1) * sc.view(n, 2, 8, 1) * q.double().view(n, 2, 8, 16)
        return w.view(-1, 256 * 1).view(n, 256)
    s = b[:, 4:16].short()
    sc = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6 << 4)], 1).double()
    mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | (s[:, 4:8] >> 6 << 4)], 1).double()
    qs = b[:, (48 if t == Q5 else 16):].view(n, 4, 32)
    q = torch.stack([qs & 15, qs >> 4], 2).view(n, 8, 32).short()
    if t == Q5:
        q += ((b[:, 16:48].short().view(n, 1, 32) >> torch.arange(8, device=b.device).view(1, 8, 1)) & 1) << 4
    return ((half(0) * sc).unsqueeze(2) * q.double() - (half(2) * mn).unsqueeze(2)).view(n, 256)


def _matrix64(t, b):
    if t is None:
        return b.double()
    out = torch.empty((b.shape[0], b.shape[1] * 256), dtype=torch.float64, device="cuda")
    for i in range(0, b.shape[0], 8192):
        out[i:i + 8192] = _dequant(t, b[i:i + 8192]).view(-1, out.shape[1])
    return out


def _rms(x, eps=1e-5):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()


def _rope_angles(n, hs, base):
    """Angles [n, hs / 2] as the model defines them: advanced in 32 bits from frequency to frequency."""
    step = np.float32(float(np.float32(base)) ** float(np.float32(-1.0 / np.float32(hs // 2))))
    a = np.arange(n, dtype=np.float32)
    out = []
    for _ in range(hs // 2):
        out.append(a)
        a = a * step
    return torch.from_numpy(np.stack(out, 1).astype(np.float64)).cuda()


class _Llama64:
    def __init__(self, c, seed):
        self.c, self.cfg = c, _config(c)
        self.types = None if c["kind"] == "generate" else LLAMAS[c["model"]][9]
        layers, self.top = _llama_tensors(c, seed)
        t = self.types or {}
        self.layers = [{k: _matrix64(t.get(k), v) if k in ROLES else v.double() for k, v in w.items()} for w in layers]

    def hidden(self, ids):
        """Normed rows in front of the classifier of sequences that each begin at position 0."""
        cfg, t = self.cfg, self.types or {}
        hs, H, G = cfg.dim // cfg.n_heads, cfg.n_heads, cfg.n_kv_heads
        lens = [len(s) for s in ids]
        every = torch.from_numpy(np.concatenate(ids).astype(np.int64)).cuda()
        x = _matrix64(t.get("emb"), self.top["emb"][every])
        ang = _rope_angles(max(lens), hs, cfg.rope_freq_base)
        cs, sn = (torch.cat([f(ang[:n]) for n in lens]).unsqueeze(1) for f in (torch.cos, torch.sin))

        def rope(v):
            a, b = (v[..., :hs // 2], v[..., hs // 2:]) if cfg.rope_is_neox else (v[..., 0::2], v[..., 1::2])
            a, b = a * cs - b * sn, a * sn + b * cs
            return torch.cat([a, b], -1) if cfg.rope_is_neox else torch.stack([a, b], -1).flatten(-2)
        for i in range(cfg.n_layers):
            w = self.layers[i % 2]
            h = _rms(x) * w["att"]
            q, k, v = (h @ w["wq"].T).view(-1, H, hs), (h @ w["wk"].T).view(-1, G, hs), (h @ w["wv"].T).view(-1, G, hs)
            q, k, at, out = rope(q), rope(k), 0, torch.empty_like(q)
            for n in lens:
                late = torch.ones((n, n), dtype=torch.bool, device="cuda").triu(1)
                for g in range(G):
                    qs = q[at:at + n, g * (H // G):(g + 1) * (H // G)].transpose(0, 1)
                    a = (qs @ k[at:at + n, g].T / math.sqrt(hs)).masked_fill_(late, -math.inf).softmax(-1)
                    out[at:at + n, g * (H // G):(g + 1) * (H // G)] = (a @ v[at:at + n, g]).transpose(0, 1)
                at += n
            x = x + out.reshape(x.shape) @ w["wo"].T
            h = _rms(x) * w["ffn"]
            x = x + (torch.nn.functional.silu(h @ w["w1"].T) * (h @ w["w3"].T)) @ w["w2"].T
        return _rms(x) * self.top["fin"].double()

    def logits(self, rows):
        if not hasattr(self, "out"):
            self.out = _matrix64((self.types or {}).get("out"), self.top["out"])
        return rows @ self.out.T


def _turn(v, pos, base, dims, halves):
    a = pos.unsqueeze(1) * base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    cs, sn, out = torch.cos(a), torch.sin(a), v.clone()
    p, q = (slice(0, dims // 2), slice(dims // 2, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out[..., p], out[..., q] = v[..., p] * cs - v[..., q] * sn, v[..., q] * cs + v[..., p] * sn
    return out


def _heads(x, n):
    return x.view(x.shape[0], n, -1).transpose(0, 1)


def _latent64(h, w, m, eps, pos):
    T, H, d, R = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
    base, dims = m["rot"]["base"], m["rot"]["dims"]
    q = _heads(h @ w["q"].T, H)
    down = h @ w["dkv"].T
    lat = _rms(down[:, :R], eps) * w["dkv.norm"]
    k, v = _heads(lat @ w["uk"].T, H), _heads(lat @ w["uv"].T, H)
    s = (q[..., :d] @ k.transpose(1, 2) + _turn(q[..., d:], pos, base, dims, False) @ _turn(down[:, R:], pos, base, dims, False).T) * m["scale"]
    s.masked_fill_(torch.ones((T, T), dtype=torch.bool, device="cuda").triu(1), -math.inf)
    s = torch.cat([s, w["sink"].view(H, 1, 1).expand(H, T, 1)], -1).softmax(-1)[..., :T]
    o = (s @ v).transpose(0, 1).reshape(T, -1)
    return (o * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def _keys64(h, w, m, eps, pos):
    T, G, d = h.shape[0], m["kv_heads"], m["dim"]
    k = (h @ w["k"].T + w["k.b"]).view(T, G, 2, d).permute(1, 2, 0, 3)
    return _turn(_rms(k, eps) * w["k.norm"], pos, m["rot"]["base"], m["rot"]["dims"], True), _heads(h @ w["v"].T + w["v.b"], G)


def _differential64(h, w, m, eps, pos, kv):
    T, H, G, d = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    k, v = kv
    q = (h @ w["q"].T + w["q.b"]).view(T, H, 2, d).permute(1, 2, 0, 3)
    q = _turn(_rms(q, eps) * w["q.norm"], pos, m["rot"]["base"], m["rot"]["dims"], True)
    late = torch.ones((T, T), dtype=torch.bool, device="cuda").triu(1)  # the chunks are longer than any of these sequences
    lam = (w["lq1"] * w["lk1"]).sum().exp() - (w["lq2"] * w["lk2"]).sum().exp() + m["diff"]
    out = []
    for i in range(H):
        g = i // (H // G)
        a = [(q[i, c] @ k[g, c].T * m["scale"]).masked_fill_(late, -math.inf).softmax(-1) @ v[g] for c in range(2)]
        out.append(_rms(a[0] - lam * a[1], eps) * (1 - m["diff"]))
    return (torch.cat(out, -1) * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def _mlstm64(h, w, m, eps):
    T, H, d, dv, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = (h @ w["q"].T).view(T, H, d) * d ** -0.5, (h @ w["k"].T).view(T, H, d), (h @ w["v"].T).view(T, H, dv)
    li = cap * torch.tanh((h @ w["i"].T + w["i.b"]) / cap)
    lf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w["f"].T + w["f.b"]) / cap))
    top = torch.zeros((T + 1, H), dtype=torch.float64, device="cuda")
    for t in range(T):
        top[t + 1] = torch.maximum(lf[t] + top[t], li[t])
    keep, add, low = (lf + top[:-1] - top[1:]).exp(), (li - top[1:]).exp(), (-top[1:]).exp()
    S, n, out = torch.zeros((H, d, dv), dtype=torch.float64, device="cuda"), torch.zeros((H, d), dtype=torch.float64, device="cuda"), torch.empty_like(v)
    for t in range(T):
        ak = add[t].unsqueeze(1) * k[t]
        S = keep[t].view(H, 1, 1) * S + ak.unsqueeze(2) * v[t].unsqueeze(1)
        n = keep[t].unsqueeze(1) * n + ak
        out[t] = (q[t].unsqueeze(1) @ S).squeeze(1) / (torch.maximum((n * q[t]).sum(-1).abs(), low[t]) + 1e-6).unsqueeze(1)
    return (_rms(out, eps).reshape(T, -1) * w["norm"] * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def _stack64(c, seed, ids):
    """Logit rows of a function of (row numbers) for one sequence."""
    raw = DESIGNS[c["model"]](c)
    W = _stack_tensors(raw, seed)
    at = {}

    def get(name):
        t = W[name]
        if t.data_ptr() not in at:
            at[t.data_ptr()] = t.double()
        return at[t.data_ptr()]
    ids = torch.from_numpy(ids.astype(np.int64)).cuda()
    pos, eps, kv = torch.arange(len(ids), dtype=torch.float64, device="cuda"), raw["norm"]["eps"], {}
    savozen = c["model"] == "savozen"
    norm = (lambda n, x: torch.tanh(get(n + ".alpha") * x) * get(n) + get(n + ".b")) if savozen else (lambda n, x: _rms(x, eps) * get(n))
    act = (lambda z: torch.nn.functional.gelu(z, approximate="tanh")) if savozen else torch.nn.functional.silu
    x = W["embed"][ids].double() * raw["embedding"]["scale"] if savozen else W["embed"][ids].double() + W["pos"][:len(ids)].double()
    for i, l in enumerate(raw["layers"]):
        p, m = f"l{i}.", l["mixer"]
        w = {k[len(p) + 4:]: get(k) for k in W if k.startswith(p + "mix.")}
        h = norm(p + "norm1", x)
        if l["type"] == "latent_attention":
            y = _latent64(h, w, m, eps, pos)
        elif l["type"] == "mlstm":
            y = _mlstm64(h, w, m, eps)
        else:
            kv[i] = kv[m["kv_from"]] if m.get("kv_from") is not None else _keys64(h, w, m, eps, pos)
            y = _differential64(h, w, m, eps, pos, kv[i])
        x = x + (y if savozen else norm(p + "norm1b", y))
        if l["mlp"]:
            h = norm(p + "norm2", x)
            y = (act(h @ get(p + "mlp.gate").T) * (h @ get(p + "mlp.up").T)) @ get(p + "mlp.down").T
            x = x + (y if savozen else norm(p + "norm2b", y))
        if savozen:
            side = raw["token_side"]["dim"]
            e = W["side.embed"][ids][:, i * side:(i + 1) * side].double()
            x = x + _rms((act(x @ get(p + "side.gate").T) * e) @ get(p + "side.proj").T, eps) * get(p + "side.norm")
    return lambda rows: norm("final.norm", x[rows]) @ get("head").T * raw.get("logit_scale", 1.0)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "product":
        t = TYPES[c["type"]]
        w = _matrix64(t, _blocks(t, c["n_out"], c["n_in"], _gen(seed, 1)))
        return torch.randn((c["cols"], c["n_in"]), generator=_gen(seed, 2), device="cuda").double() @ w.T
    if kind == "batch":
        ids, late = _batch_script(c, seed)
        own = [s[d:] for s, d in zip(ids, late)]
        if c["model"] in DESIGNS:
            return dict(logits=torch.cat([_stack64(c, seed, s)([-1]) for s in own])) if c["seqs"] * c["layers"] <= 100 else None
        m = _Llama64(c, seed)
        ends = np.cumsum([len(s) for s in own])
        rows = m.hidden(own)
        steps = [m.logits(rows[ends - c["steps"] + i]) for i in range(c["steps"])]
        return dict(tokens=torch.stack([s.argmax(-1) for s in steps]), logits=steps[-1])
    ids = _ids(seed, c.get("prompt", 0) + c.get("past", 0) + c.get("tokens", 0) + c.get("steps", 0), _vocab(c))
    if kind == "portion":
        return dict(logits=_stack64(c, seed, ids)(_wanted(c)))
    if kind == "trace":
        return dict(logits=_stack64(c, seed, ids)(list(range(c["tokens"] - 1, len(ids)))))
    m = _Llama64(c, seed)
    if kind == "generate":
        for i in range(len(ids), c["positions"]):
            ids = np.append(ids, m.logits(m.hidden([ids])[-1]).argmax().item())
        last = m.logits(m.hidden([ids]))
        return dict(tokens=last.argmax(-1), logits=last[-1])
    if kind == "prefill":
        last = m.logits(m.hidden([ids])[-1])
        return dict(next=last.argmax(), logits=last)
    last = m.logits(m.hidden([ids])[-c["steps"]:])
    return dict(logits=last[-1]) if c["temperature"] else dict(tokens=last.argmax(-1), logits=last[-1])
