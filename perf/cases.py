"""The work that users of this library have it do, as cases that can be timed and compared.

A case goes through the public entry points alone (``Engine.step``, ``new_sequence`` / ``free_sequence`` / ``truncate`` and
``generate``) on models with random weights: the library has no trained checkpoint of its own, and a step's work does not
depend on the weights' values, except for which experts a routed layer's tokens choose (see ``_design_weights``).

Kinds of cases (``"kind"``):

* ``decode``: one token for each of some sequences that hold ``context`` positions: the step that generation repeats. The
  sequences are rolled back afterwards, so every pass is the same step.
* ``prompt``: the prompts of a batch of requests in one step, from empty sequences.
* ``serve``: prompts in one step and then ``steps`` steps of one token each: what ``generate`` does with a batch, with the
  tokens given instead of sampled, for the designs whose sequences cannot be rolled back (recurrent states, windows).
* ``generate``: the whole generation loop with sampling, tokens in and tokens out.

Models (``"model"``): ``8b`` has the layer sizes and the vocabulary of Apertus-8B (hidden 4,096, 32 / 8 heads of 128, feed-forward
21,504, vocabulary 131,072), with 16 of its 32 layers in bfloat16 and 8 of them in 32-bit, which keeps several of them on one GPU;
``mid`` is Apertus at hidden 2,048 with 16 / 4 heads of 64, 8 layers; ``vogilix``, ``zudepel`` and ``fasodra`` are those designs at width
2,048 with 8 layers; ``tiny`` is the second tiny configuration of the tests.
"""
import math
import zlib

import torch

F64 = torch.float64


# ---------------------------------------------------------------------------------------------------- models
def _apertus(layers, hidden, heads, kv_heads, head_dim, inter, vocab, positions):
    return {"architectures": ["ApertusForCausalLM"], "model_type": "apertus", "num_hidden_layers": layers, "hidden_size": hidden,
            "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": head_dim, "intermediate_size": inter,
            "vocab_size": vocab, "rope_theta": 12000000.0,
            "rope_scaling": {"rope_type": "llama3", "factor": 8.0, "original_max_position_embeddings": 8192, "low_freq_factor": 1.0,
                             "high_freq_factor": 4.0},
            "rms_norm_eps": 1e-5, "qk_norm": True, "tie_word_embeddings": False, "hidden_act": "xielu",
            "max_position_embeddings": positions, "attention_bias": False, "mlp_bias": False}


_TINY = {"architectures": ["ApertusForCausalLM"], "model_type": "apertus", "num_hidden_layers": 3, "hidden_size": 96,
         "num_attention_heads": 6, "num_key_value_heads": 3, "head_dim": 32, "intermediate_size": 320, "vocab_size": 512,
         "rope_theta": 12000000.0,
         "rope_scaling": {"rope_type": "llama3", "factor": 8.0, "original_max_position_embeddings": 64, "low_freq_factor": 1.0,
                          "high_freq_factor": 4.0},
         "rms_norm_eps": 1e-6, "qk_norm": True, "tie_word_embeddings": True, "hidden_act": "xielu", "max_position_embeddings": 1024,
         "attention_bias": False, "mlp_bias": False}
POSITIONS = 4096            # of the designs' models
WIDTH, VOCAB, LAYERS = 2048, 32768, 8


def _vogilix():
    mixer = {"dim": 64, "heads": 16, "kv_rank": 128, "mask": {"size": 1024}, "q_rank": 768, "scale": 64 ** -0.5, "vdim": 64}
    moe = {"expert": {"ff": 1024, "limit": 7.0}, "kind": "moe", "router": {"experts": 32, "top": 4}, "shared": {"ff": 2048, "limit": 7.0}}
    return {"architecture": "Vogilix", "vocab": VOCAB, "width": WIDTH, "max_positions": POSITIONS, "norm": {"eps": 1e-6},
            "residual_mult": 0.5, "token_side": {"dim": 64},
            "layers": [{"mixer": mixer, "mlp": {"ff": 8192, "kind": "dense"} if i == 0 else moe, "type": "latent_attention"}
                       for i in range(LAYERS)]}


def _zudepel():
    decay = [math.exp(-2.0 ** (-8.0 * (h + 1) / 16)) for h in range(16)]
    moe = {"expert": {"ff": 1024}, "kind": "moe", "router": {"experts": 32, "groups": {"count": 4, "keep": 2}, "identity": 4, "top": 4},
           "shared": {"ff": 2048}}
    layers = []
    for i in range(LAYERS):
        mlp = {"ff": 8192, "kind": "dense"} if i == 0 else moe
        if i % 2 == 0:
            layers.append({"mixer": {"decay": decay, "dim": 128, "heads": 16, "vdim": 128}, "mlp": mlp, "type": "lightning"})
            continue
        m = {"conv": 4, "dim": 128, "heads": 16, "kv_heads": 4, "rot": {"base": 10000.0, "dims": 64}, "scale": 128 ** -0.5, "vdim": 128}
        if i % 4 == 3:
            m["kv_from"] = i - 2
        layers.append({"mixer": m, "mlp": mlp, "type": "attention"})
    return {"architecture": "Zudepel", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": 1e-6}, "layers": layers}


def _fasodra():
    moe = {"expert": {"ff": 1024}, "kind": "moe", "router": {"experts": 32, "top": 4}}
    base = {"dim": 128, "heads": 16, "kv_heads": 4, "scale": 128 ** -0.5, "vdim": 128}
    left = {**base, "rot": {"base": 10000.0, "dims": 64}}
    kinds = [("attention", {**base, "bias_max": 2048, "mask": {"size": 1024}}),
             ("parallel_2", {"left": left, "right": {"conv": 4, "dim": 128, "heads": 16, "kv_heads": 8, "vdim": 128}}),
             ("attention", {**base, "bias_max": 2048, "mask": {"size": 1024}}),
             ("parallel", {"left": left, "left_scale": 1.0, "right": {"dim": 64, "heads": WIDTH // 64}, "right_scale": 1.0})]
    return {"architecture": "Fasodra", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": 1e-6}, "residual_mult": 0.5, "streams": 2,
            "layers": [{"mixer": kinds[i % 4][1], "mlp": moe, "type": kinds[i % 4][0]} for i in range(LAYERS)]}


DESIGNS = {"vogilix": _vogilix, "zudepel": _zudepel, "fasodra": _fasodra}


def _config(case):
    model = case["model"]
    if model in DESIGNS:
        return DESIGNS[model]()
    if model == "tiny":
        return dict(_TINY)
    positions = -(-(max(_lengths(case)) + 65) // 1024) * 1024
    if model == "8b":
        return _apertus(16 if case["dtype"] == "bfloat16" else 8, 4096, 32, 8, 128, 21504, 131072, positions)
    return _apertus(8, 2048, 16, 4, 64, 9216, 32768, positions)


# ---------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # The smallest call: a short batch generated with sampling by a model of a few layers. Launches and host time count.
        {"name": "tiny-generate", "kind": "generate", "model": "tiny", "dtype": "float32", "lengths": "1,4,17,33,70", "steps": 12},
        # One user's chat: a token at a time after a thousand positions. Reading the weights once is the floor.
        {"name": "8b-decode-1", "kind": "decode", "model": "8b", "dtype": "bfloat16", "lengths": "1023"},
        # A small and a large batch of requests in the middle of their answers.
        {"name": "8b-decode-8", "kind": "decode", "model": "8b", "dtype": "bfloat16", "lengths": "1023*8"},
        {"name": "8b-decode-64", "kind": "decode", "model": "8b", "dtype": "bfloat16", "lengths": "1023*64"},
        # Documents of very unequal lengths being answered together: the cache is most of what a step reads.
        {"name": "8b-decode-long", "kind": "decode", "model": "8b", "dtype": "bfloat16", "lengths": "15873,9001,3352,511,77"},
        # A long prompt, and a batch of short, unequal ones (a few questions that arrive together).
        {"name": "8b-prompt-2048", "kind": "prompt", "model": "8b", "dtype": "bfloat16", "lengths": "2048"},
        {"name": "8b-prompts-ragged", "kind": "prompt", "model": "8b", "dtype": "bfloat16", "lengths": "5,37,130,411,700"},
        # The true 32-bit path, which users take to check a model: a batch being decoded, and prompts.
        {"name": "8b-decode-8-float32", "kind": "decode", "model": "8b", "dtype": "float32", "lengths": "255,31,97,130,255,12,201,64"},
        {"name": "8b-prompts-float32", "kind": "prompt", "model": "8b", "dtype": "float32", "lengths": "300,129,83"},
        # Designs with latent attention, routed experts, linear attention, delta rule and time mixing: batches of requests from
        # the prompts on, and a long prompt with the start of its answer.
        {"name": "vogilix-serve", "kind": "serve", "model": "vogilix", "dtype": "bfloat16", "lengths": "300,41,128,77,19,250,64,103", "steps": 16},
        {"name": "zudepel-serve-long", "kind": "serve", "model": "zudepel", "dtype": "bfloat16", "lengths": "2048", "steps": 4},
        {"name": "fasodra-serve", "kind": "serve", "model": "fasodra", "dtype": "bfloat16", "lengths": "1500,333,64,7", "steps": 16},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "prompt", "decode32", "prompt32", "serve", "serve", "serve", "generate"])
    apertus = rng.choice(["8b", "8b", "mid"])
    text = lambda lengths: ",".join(str(n) for n in lengths)                                                  # noqa: E731
    if kind == "decode":
        batch = _log(rng, 1, 64)
        most = min(16000, 66000 // batch)
        top = _log(rng, 64, most)
        lengths = [top] * batch if rng.random() < 0.5 else [_log(rng, 16, top) for _ in range(batch)]
        return {"kind": "decode", "model": apertus, "dtype": "bfloat16", "lengths": text(lengths)}
    if kind == "prompt":
        count = rng.choice([1, 1, 1, 2, 3, 5, 8])
        lengths = [_log(rng, 3 if count > 1 else 24, 2048 // count) for _ in range(count)]
        return {"kind": "prompt", "model": apertus, "dtype": "bfloat16", "lengths": text(lengths)}
    if kind == "decode32":
        batch = _log(rng, 1, 32)
        return {"kind": "decode", "model": apertus, "dtype": "float32", "lengths": text(_log(rng, 8, max(16, min(512, 1200 // batch))) for _ in range(batch))}
    if kind == "prompt32":
        count = rng.choice([1, 1, 2, 4])
        return {"kind": "prompt", "model": apertus, "dtype": "float32", "lengths": text(_log(rng, 3, 512 // count) for _ in range(count))}
    if kind == "serve":
        model = rng.choice(sorted(DESIGNS))
        count = rng.choice([1, 1, 2, 4, 8])
        lengths = [_log(rng, 3, 2048 // count) for _ in range(count)]
        return {"kind": "serve", "model": model, "dtype": "bfloat16", "lengths": text(lengths), "steps": rng.choice([2, 4, 8, 16])}
    count = rng.randint(1, 8)
    return {"kind": "generate", "model": "tiny", "dtype": "float32", "lengths": text(_log(rng, 1, 90) for _ in range(count)),
            "steps": rng.randint(4, 16)}


def _lengths(case):
    out = []
    for part in case["lengths"].split(","):
        n, _, times = part.partition("*")
        out += [int(n)] * int(times or 1)
    return out


def _tokens(case, seed, vocab):
    """(prompts, the tokens after them: one list per later step)."""
    g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    lengths = _lengths(case)
    ids = torch.randint(0, vocab, (sum(lengths),), generator=g).tolist()
    prompts, at = [], 0
    for n in lengths:
        prompts.append(ids[at:at + n])
        at += n
    steps = 1 if case["kind"] == "decode" else case.get("steps", 0) if case["kind"] == "serve" else 0
    return prompts, [torch.randint(0, vocab, (len(lengths),), generator=g).tolist() for _ in range(steps)]


# ---------------------------------------------------------------------------------------------------- weights
class _Maker:
    """Random tensors on the GPU, each from the seed and its own name."""

    def __init__(self, seed):
        self.seed, self.out = int(seed), {}

    def normal(self, name, shape, std, mean=0.0):
        g = torch.Generator(device="cuda").manual_seed((zlib.crc32(name.encode()) + 1000003 * self.seed) & 0x7FFFFFFF)
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        flat, step = t.view(-1), 1 << 27                 # bounds the 32-bit scratch of the large tables
        for a in range(0, flat.numel(), step):
            n = min(step, flat.numel() - a)
            flat[a:a + n] = torch.randn(n, generator=g, device="cuda").mul_(std).add_(mean)
        self.out[name] = t
        return t

    def matrix(self, name, rows, cols):
        return self.normal(name, (rows, cols), cols ** -0.5)

    def gain(self, name, size):
        return self.normal(name, (size,), 0.1, 1.0)


def _apertus_weights(cfg, seed):
    m = _Maker(seed)
    H, I, D = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    nq, nkv, V = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["vocab_size"]
    lin = lambda name, rows, cols: m.normal(name, (rows, cols), 0.02)                                         # noqa: E731
    one = lambda name, size: m.normal(name, (size,), 0.02, 1.0)                                               # noqa: E731
    lin("model.embed_tokens.weight", V, H)
    if not cfg["tie_word_embeddings"]:
        lin("lm_head.weight", V, H)
    one("model.norm.weight", H)
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        one(p + "attention_layernorm.weight", H)
        one(p + "feedforward_layernorm.weight", H)
        lin(p + "self_attn.q_proj.weight", nq * D, H)
        lin(p + "self_attn.k_proj.weight", nkv * D, H)
        lin(p + "self_attn.v_proj.weight", nkv * D, H)
        lin(p + "self_attn.o_proj.weight", H, nq * D)
        one(p + "self_attn.q_norm.weight", D)
        one(p + "self_attn.k_norm.weight", D)
        lin(p + "mlp.up_proj.weight", I, H)
        lin(p + "mlp.down_proj.weight", H, I)
        for name in ("alpha_p", "alpha_n"):
            m.normal(p + "mlp.act_fn." + name, (1,), 0.05, math.log(math.exp(0.8) - 1))
        m.out[p + "mlp.act_fn.beta"] = torch.full((), 0.5, dtype=torch.bfloat16, device="cuda")
        m.out[p + "mlp.act_fn.eps"] = torch.full((), -1e-6, dtype=torch.bfloat16, device="cuda")
    return m.out


def _design_weights(cfg, seed):
    """Weights of the three designs. A trained router is seldom in two minds; a random one always is, and which expert a near tie
    goes to would depend on the last bit of its input. So every token leans towards ``top`` experts of every routed layer: its
    embedding holds a multiple of those experts' router rows. Which experts those are is random, per token and layer."""
    m = _Maker(seed)
    W, V, kind = cfg["width"], cfg["vocab"], cfg["architecture"]
    embed = torch.empty((V, W), dtype=torch.float32, device="cuda").normal_(generator=torch.Generator(device="cuda").manual_seed(int(seed) + 11))
    m.matrix("head", V, W)
    norm = (lambda name, size: m.normal(name, (size,), 0.1)) if kind == "Vogilix" else m.gain
    names = ["final.norm"] + ["l%d.norm%d" % (i, k) for i in range(len(cfg["layers"])) for k in ((1, 2) if kind != "Zudepel" else (1,))]
    for name in names:
        norm(name, W)
        if kind == "Fasodra":
            m.normal(name + ".b", (W,), 0.1)
    if kind == "Vogilix":
        side = cfg["token_side"]["dim"]
        m.normal("pos", (cfg["max_positions"], W), 0.5)
        m.normal("side.embed", (V, side * len(cfg["layers"])), 1.0)
    for i, layer in enumerate(cfg["layers"]):
        L = "l%d." % i
        _mixer_weights(m, layer["type"], layer["mixer"], L + "mix.", W, kind)
        mlp, p = layer["mlp"], L + "mlp."
        if kind == "Vogilix":
            m.matrix(L + "side.gate", side, W)
            m.matrix(L + "side.proj", W, side)
            m.gain(L + "side.norm", W)
        if kind == "Fasodra":
            for q in ("hc1.", "hc2."):
                m.normal(L + q + "in", (2,), 0.1, 0.5)
                m.normal(L + q + "out", (2,), 0.2, 1.0)
                m.normal(L + q + "mix", (2, 2), 0.15, 0.5)
        if mlp["kind"] == "dense":
            if kind == "Zudepel":
                m.matrix(p + "gate", mlp["ff"], W)
            m.matrix(p + "up", mlp["ff"], W)
            m.matrix(p + "down", W, mlp["ff"])
            continue
        r, ff = mlp["router"], mlp["expert"]["ff"]
        total = r["experts"] + r.get("identity", 0)
        rows = m.normal(p + "router", (total, W), (2.0 if kind != "Vogilix" else 0.5) * W ** -0.5)
        unit = rows.float() / rows.float().norm(dim=1, keepdim=True)
        g = torch.Generator(device="cuda").manual_seed(int(seed) * 131 + i)
        score = torch.rand((V, total), generator=g, device="cuda")
        if r.get("groups"):                                # the chosen experts lie in the groups that are kept
            count, keep = r["groups"]["count"], r["groups"]["keep"]
            of = torch.rand((V, count), generator=g, device="cuda").topk(keep, 1).indices
            kept = torch.zeros((V, count), dtype=torch.bool, device="cuda").scatter_(1, of, True)
            per = score.view(V, count, total // count)
            first = torch.zeros_like(per).scatter_(2, per.max(2, keepdim=True).indices, 1.0)     # one in each kept group
            score = ((per + first) * kept[:, :, None]).view(V, total)
        chosen = score.topk(r["top"], 1).indices
        for j in range(r["top"]):
            embed += 10.0 * unit[chosen[:, j]]
        if kind == "Zudepel":
            m.normal(p + "correction", (total,), 0.02)
            m.matrix(p + "shared.sg", 1, W)
        parts = ("up", "down") if kind == "Fasodra" else ("gate", "up", "down")
        units = [("e%d." % e, ff) for e in range(r["experts"])] + ([("shared.", mlp["shared"]["ff"])] if mlp.get("shared") else [])
        for name, size in units:
            for part in parts:
                m.matrix(p + name + part, W if part == "down" else size, size if part == "down" else W)
    m.out["embed"] = embed.to(torch.bfloat16)
    return m.out


def _mixer_weights(m, kind, x, p, W, design):
    if kind == "latent_attention":
        H, D, V = x["heads"], x["dim"], x["vdim"]
        for name, rows, cols in (("dq", x["q_rank"], W), ("uq", H * D, x["q_rank"]), ("dkv", x["kv_rank"], W), ("uk", H * D, x["kv_rank"]),
                                 ("uv", H * V, x["kv_rank"]), ("o", W, H * V)):
            m.matrix(p + name, rows, cols)
        m.gain(p + "dq.norm", x["q_rank"])
        m.gain(p + "dkv.norm", x["kv_rank"])
    elif kind == "lightning":
        H, D, V = x["heads"], x["dim"], x["vdim"]
        for name, rows, cols in (("q", H * D, W), ("k", H * D, W), ("v", H * V, W), ("g", H * V, W), ("o", W, H * V)):
            m.matrix(p + name, rows, cols)
        m.gain(p + "norm", H * V)
    elif kind == "attention" or kind == "left":
        H, G, D, V = x["heads"], x["kv_heads"], x["dim"], x["vdim"]
        m.matrix(p + "o", W, H * V)
        if design == "Zudepel":
            m.matrix(p + "g", H * V, W)
            m.normal(p + "sink", (H,), 1.0)
        for name, rows in (("q", H * D), ("k", G * D), ("v", G * V)):
            if name != "q" and x.get("kv_from") is not None:
                continue
            m.matrix(p + name, rows, W)
            m.normal(p + name + ".b", (rows,), 0.1)
            if x.get("conv"):
                m.normal(p + name + ".conv", (rows, x["conv"]), 0.3, 0.25)
            if design == "Zudepel" and name != "v":
                m.gain(p + name + ".norm", rows)
        if design == "Fasodra" and kind == "attention":
            m.normal(p + "rel", (16, H), 1.0)
    elif kind == "parallel":
        _mixer_weights(m, "left", x["left"], p + "left.", W, design)
        m.matrix(p + "left.g", x["left"]["heads"], W)
        r, q = x["right"], p + "right."
        size = r["heads"] * r["dim"]
        for s in "rkvgw":
            m.normal(q + "mu." + s, (W,), 0.25, 0.5)
        for s in "rkvg":
            m.matrix(q + s, size, W)
        m.matrix(q + "w1", 64, W)
        m.normal(q + "w2", (size, 64), 0.5 * 64 ** -0.5)
        m.normal(q + "w0", (size,), 1.0, -2.5)
        m.normal(q + "u", (r["heads"], r["dim"]), 0.5)
        m.gain(q + "norm", size)
        m.matrix(q + "o", W, size)
    elif kind == "parallel_2":
        _mixer_weights(m, "left", x["left"], p + "left.", W, design)
        m.gain(p + "left.q.norm", x["left"]["dim"])
        m.gain(p + "left.k.norm", x["left"]["dim"])
        r, q = x["right"], p + "right."
        H, G, D, V = r["heads"], r["kv_heads"], r["dim"], r["vdim"]
        for name, rows in (("q", G * D), ("k", G * D), ("v", H * V)):
            m.matrix(q + name, rows, W)
            m.normal(q + name + ".conv", (rows, r["conv"]), 0.3, 0.25)
        m.matrix(q + "g", H * V, W)
        m.matrix(q + "b", H, W)
        m.matrix(q + "a", H, W)
        m.normal(q + "A_log", (H,), 0.5)
        m.normal(q + "dt_bias", (H,), 1.0, -2.0)
        m.gain(q + "norm", V)
        m.matrix(q + "o", W, H * V)
        m.gain(p + "left.out", W)
        m.gain(p + "right.out", W)


def _weights(cfg, seed):
    return _design_weights(cfg, seed) if "architecture" in cfg else _apertus_weights(cfg, seed)


# ---------------------------------------------------------------------------------------------------- the call
def prepare(case, seed):
    """A loaded model, the requests' tokens, and for ``decode`` sequences that hold their contexts."""
    import tileinfer_b200 as ti
    from tileinfer_b200.config import config_from_dict
    raw = _config(case)
    lengths = _lengths(case)
    vocab = raw.get("vocab") or raw["vocab_size"]
    prompts, later = _tokens(case, seed, vocab)
    room = sum(-(-(n + case.get("steps", 1) + 2) // 64) * 64 for n in lengths)
    engine = ti.Engine(config_from_dict(raw), _weights(raw, seed), dtype=case["dtype"], max_context=max(lengths) + 64, max_seqs=max(8, len(lengths)),
                       max_tokens=max(1024, room))
    state = {"case": case, "engine": engine, "prompts": prompts, "later": later, "lengths": lengths, "seed": int(seed)}
    if case["kind"] == "decode":
        state["slots"] = [engine.new_sequence() for _ in prompts]
        engine.step(list(zip(state["slots"], prompts)))
    return state


def run(state):
    import tileinfer_b200 as ti
    case, engine = state["case"], state["engine"]
    if case["kind"] == "generate":
        tokens = ti.generate(engine, state["prompts"], max_new_tokens=case["steps"], sampling=ti.SamplingParams(temperature=0.8, top_k=50, top_p=0.95),
                             stop_ids=[], seed=state["seed"])
        return torch.tensor(tokens)
    if case["kind"] == "decode":
        slots = state["slots"]
        logits = engine.step([(s, [t]) for s, t in zip(slots, state["later"][0])])
        for s, n in zip(slots, state["lengths"]):
            engine.truncate(s, n)
        return logits
    slots = [engine.new_sequence() for _ in state["prompts"]]
    logits = [engine.step(list(zip(slots, state["prompts"])))]
    for tokens in state["later"]:
        last = engine.step([(s, [t]) for s, t in zip(slots, tokens)])
    if state["later"]:
        logits.append(last)
    for s in slots:
        engine.free_sequence(s)
    return logits


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    cfg, lengths = _config(case), _lengths(case)
    B, size = len(lengths), 2 if case["dtype"] == "bfloat16" else 4
    steps = case.get("steps", 0)
    if "architecture" not in cfg:
        H, I, D, L = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"], cfg["num_hidden_layers"]
        nq, nkv, V = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["vocab_size"]
        layer, head = H * (nq + 2 * nkv) * D + nq * D * H + 2 * H * I, V * H
        kv = 2 * nkv * D * L * size                       # per position
        score = 4 * nq * D * L                            # multiply-adds times two, per (query, key) pair

        def step(queries, cached):
            pairs = sum(c * q + q * (q + 1) // 2 for q, c in zip(queries, cached))
            n = sum(queries)
            return {"bytes": (L * layer + head) * size + kv * (n + sum(cached)) + 4 * V * B,
                    "flops": 2 * n * L * layer + 2 * B * head + score * pairs}
    else:
        W, V, kind = cfg["width"], cfg["vocab"], cfg["architecture"]
        fixed = expert = active = kv = state = score = 0
        for layer in cfg["layers"]:
            x, mlp, kind_ = layer["mixer"], layer["mlp"], layer["type"]
            if kind_ == "latent_attention":
                H, D, r, c = x["heads"], x["dim"], x["q_rank"], x["kv_rank"]
                fixed += W * (r + c) + H * D * (r + 2 * c) + H * D * W + 2 * cfg["token_side"]["dim"] * W
                kv, score = kv + c * 2, score + 4 * H * c
            elif kind_ == "lightning":
                H, D = x["heads"], x["dim"]
                fixed, state, score = fixed + 5 * W * H * D, state + 8 * H * D * D, score
                active += 2 * H * D * D
            else:
                a = x if kind_ == "attention" else x["left"]
                fixed += 2 * W * a["heads"] * a["dim"] + (0 if a.get("kv_from") is not None else 2 * W * a["kv_heads"] * a["dim"])
                fixed += W * a["heads"] * a["dim"] if kind == "Zudepel" else 0
                kv, score = kv + (0 if a.get("kv_from") is not None else 4 * a["kv_heads"] * a["dim"]), score + 4 * a["heads"] * a["dim"]
                if kind_ != "attention":
                    r = x["right"]
                    H, D = r["heads"], r["dim"]
                    fixed += W * D * (4 * H if kind_ == "parallel_2" else 5 * H)
                    state, active = state + 8 * H * D * D, active + 3 * H * D * D
            if mlp["kind"] == "dense":
                fixed += (3 if kind == "Zudepel" else 2) * W * mlp["ff"]
            else:
                parts = 2 if kind == "Fasodra" else 3
                expert += parts * W * mlp["expert"]["ff"] * mlp["router"]["experts"]
                active += parts * W * mlp["expert"]["ff"] * mlp["router"]["top"]
                fixed += parts * W * mlp["shared"]["ff"] if mlp.get("shared") else 0

        def step(queries, cached):
            n = sum(queries)
            share = 1 - (1 - 4 / 32) ** n                 # experts that some token of the step takes
            seen = 1 << 30 if kind == "Zudepel" else 1024    # the windows and chunks
            pairs = sum(sum(min(seen, c + i + 1) for i in range(q)) for q, c in zip(queries, cached))
            return {"bytes": 2 * (fixed + share * expert + V * W) + kv * (n + sum(min(seen, c) for c in cached)) + 2 * state * B + 4 * V * B,
                    "flops": 2 * n * (fixed + active) + 2 * B * V * W + score * pairs}
    if case["kind"] == "decode":
        return step([1] * B, lengths)
    total = step(lengths, [0] * B)
    for k in range(steps if case["kind"] == "serve" else steps - 1 if case["kind"] == "generate" else 0):
        one = step([1] * B, [n + k for n in lengths])
        total = {"bytes": total["bytes"] + one["bytes"], "flops": total["flops"] + one["flops"]}
    return total


def tolerance(case):
    """From the distance to 64-bit arithmetic, measured at these cases: 1.7e-2 with bfloat16 activations through 16 Apertus layers, 5e-3
    through the designs' 8, 7e-6 with 32-bit sums. Two correct implementations may be that far off in different directions. Sampled
    tokens are the same unless a draw falls within rounding of a boundary."""
    if case["kind"] == "generate":
        return {"rel": 0.0, "differ": 0.01}
    if case["dtype"] == "float32":
        return {"rel": 3e-5, "max": 5e-4}
    return {"rel": 0.03, "max": 0.5}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """The logits in plain torch and 64-bit arithmetic on the same weights: every sequence alone, nothing cached."""
    lengths = _lengths(case)
    if case["kind"] == "generate" or sum(lengths) > 9000 or max(lengths) > 4500:
        return None
    cfg = _config(case)
    prompts, later = _tokens(case, seed, cfg.get("vocab") or cfg["vocab_size"])
    full = [p + [t[b] for t in later] for b, p in enumerate(prompts)]
    wanted = [[len(s) - 1] if case["kind"] == "decode" or not later else [len(p) - 1, len(s) - 1] for p, s in zip(prompts, full)]
    weights = _weights(cfg, seed)
    with torch.no_grad():
        rows = _exact_design(cfg, weights, full, wanted) if "architecture" in cfg else _exact_apertus(cfg, weights, full, wanted)
    if case["kind"] == "decode":
        return rows[:, 0]
    return [rows[:, k].contiguous() for k in range(rows.shape[1])]


def _mm(x, w):
    return x @ w.to(F64).t()


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _inverse_frequencies(cfg):
    """In 32-bit, as the architecture defines them, with the llama3 scaling."""
    D, s = cfg["head_dim"], cfg["rope_scaling"]
    inv = 1.0 / (torch.tensor(cfg["rope_theta"], dtype=torch.float32) ** (torch.arange(0, D, 2, dtype=torch.float32) / D))
    factor, low, high, old = (torch.tensor(float(s[k]), dtype=torch.float32)
                              for k in ("factor", "low_freq_factor", "high_freq_factor", "original_max_position_embeddings"))
    wave = 2.0 * torch.tensor(math.pi, dtype=torch.float32) / inv
    smooth = (old / wave - low) / (high - low)
    mid = (1 - smooth) * inv / factor + smooth * inv
    return torch.where(wave < old / high, inv, torch.where(wave > old / low, inv / factor, mid))


def _attend(q, k, v, scale, visible=None, bias=None, sink=None):
    """q [n, heads, d], k [n, groups, d], v [n, groups, e]; all positions at once, one head after the other."""
    n, H, _ = q.shape
    rep = H // k.shape[1]
    if visible is None:
        visible = torch.ones((n, n), dtype=torch.bool, device=q.device).tril_()
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].t()) * scale
        if bias is not None:
            s = s + bias(h)
        s = s.masked_fill(~visible, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :n] @ v[:, h // rep])
    return torch.stack(out, 1)


def _exact_apertus(cfg, W, sequences, wanted):
    D, eps = cfg["head_dim"], cfg["rms_norm_eps"]
    ids = torch.tensor([t for s in sequences for t in s], device="cuda")
    pos = torch.tensor([i for s in sequences for i in range(len(s))], dtype=torch.float32)
    angle = (pos[:, None] * _inverse_frequencies(cfg)[None, :]).to("cuda").to(F64)
    cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]

    def turn(x):
        u, v = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)

    x = W["model.embed_tokens.weight"][ids].to(F64)
    for i in range(cfg["num_hidden_layers"]):
        w = lambda name: W["model.layers.%d.%s" % (i, name)]                                                  # noqa: E731
        h = _rms(x, eps) * w("attention_layernorm.weight").to(F64)
        q, k, v = (_mm(h, w("self_attn.%s_proj.weight" % s)).view(len(ids), -1, D) for s in "qkv")
        q = turn(_rms(q, eps) * w("self_attn.q_norm.weight").to(F64))
        k = turn(_rms(k, eps) * w("self_attn.k_norm.weight").to(F64))
        o, a = [], 0
        for s in sequences:
            b = a + len(s)
            o.append(_attend(q[a:b], k[a:b], v[a:b], D ** -0.5))
            a = b
        x = x + _mm(torch.cat(o).reshape(len(ids), -1), w("self_attn.o_proj.weight"))
        h = _rms(x, eps) * w("feedforward_layernorm.weight").to(F64)
        u = _mm(h, w("mlp.up_proj.weight"))
        beta, low = w("mlp.act_fn.beta").to(F64), w("mlp.act_fn.eps").to(F64)
        p, n = (torch.log1p(torch.exp(w("mlp.act_fn.alpha_" + s).to(F64))) for s in "pn")
        u = torch.where(u > 0, p * u * u + beta * u, (torch.expm1(torch.minimum(u, low)) - u) * (beta + n) + beta * u)
        x = x + _mm(u, w("mlp.down_proj.weight"))
    at, rows = 0, []
    for s, wants in zip(sequences, wanted):
        rows += [at + j for j in wants]
        at += len(s)
    h = _rms(x[rows], eps) * W["model.norm.weight"].to(F64)
    head = W["model.embed_tokens.weight"] if cfg["tie_word_embeddings"] else W["lm_head.weight"]
    return _mm(h, head).view(len(sequences), -1, head.shape[0])


def _rotate(x, dims, base):
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / dims)
    a = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * f[None, :]
    cos, sin = a.cos()[:, None, :], a.sin()[:, None, :]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., dims:]], -1)


def _conv(u, c):
    y, taps = torch.zeros_like(u), c.shape[1]
    for j in range(taps):
        shift = taps - 1 - j
        if shift < u.shape[0]:
            y[shift:] += c[:, j].to(F64) * u[:u.shape[0] - shift]
    return y


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu_tanh(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _window(n, size):
    i = torch.arange(n, device="cuda")
    d = i[:, None] - i[None, :]
    return (d >= 0) & (d < size)


def _mix(kind, design, h, W, p, x, eps, kept, layer):
    n = h.shape[0]
    if kind == "latent_attention":
        c = _rms(_mm(h, W[p + "dkv"]), eps) * W[p + "dkv.norm"].to(F64)
        q = _mm(_rms(_mm(h, W[p + "dq"]), eps) * W[p + "dq.norm"].to(F64), W[p + "uq"]).view(n, x["heads"], -1)
        k, v = (_mm(c, W[p + s]).view(n, x["heads"], -1) for s in ("uk", "uv"))
        return _mm(_attend(q, k, v, x["scale"], _window(n, x["mask"]["size"])).reshape(n, -1), W[p + "o"])
    if kind == "lightning":
        q, k, v = (_silu(_mm(h, W[p + s])).view(n, x["heads"], -1) for s in "qkv")
        decay = torch.tensor(x["decay"], dtype=F64, device="cuda")[:, None, None]
        S, o = torch.zeros((x["heads"], x["dim"], x["vdim"]), dtype=F64, device="cuda"), []
        for t in range(n):
            S = decay * S + k[t][:, :, None] * v[t][:, None, :]
            o.append(torch.bmm(q[t][:, None, :], S)[:, 0])
        y = _rms(torch.stack(o).reshape(n, -1), eps) * W[p + "norm"].to(F64)
        return _mm(y * torch.sigmoid(_mm(h, W[p + "g"])), W[p + "o"])
    if kind == "attention" and design == "Zudepel":
        def inputs(name):
            u = _conv(_mm(h, W[p + name]) + W[p + name + ".b"].to(F64), W[p + name + ".conv"])
            if name != "v":
                u = _rms(u, eps) * W[p + name + ".norm"].to(F64)
            u = u.view(n, -1, x["dim"])
            return u if name == "v" else _rotate(u, x["rot"]["dims"], x["rot"]["base"])
        if x.get("kv_from") is None:
            kept[layer] = (inputs("k"), inputs("v"))
        k, v = kept[x["kv_from"] if x.get("kv_from") is not None else layer]
        o = _attend(inputs("q"), k, v, x["scale"], sink=W[p + "sink"].to(F64)).reshape(n, -1)
        return _mm(o * torch.sigmoid(_mm(h, W[p + "g"])), W[p + "o"])
    if kind in ("attention", "left"):
        q, k, v = ((_mm(h, W[p + s]) + W[p + s + ".b"].to(F64)).view(n, -1, x["dim"]) for s in "qkv")
        if kind == "left":
            if p + "q.norm" in W:
                q, k = _rms(q, eps) * W[p + "q.norm"].to(F64), _rms(k, eps) * W[p + "k.norm"].to(F64)
            q, k = (_rotate(u, x["rot"]["dims"], x["rot"]["base"]) for u in (q, k))
            o = _attend(q, k, v, x["scale"])
            if p + "g" in W:
                o = o * torch.sigmoid(_mm(h, W[p + "g"]))[:, :, None]
            return _mm(o.reshape(n, -1), W[p + "o"])
        size, rel = x["mask"]["size"], W[p + "rel"].to(F64)
        rows, half, far = rel.shape[0], rel.shape[0] // 2, x["bias_max"]
        row = [d if d < half else min(rows - 1, half + int(math.floor(math.log(d / half) / math.log(far / half) * (rows - half)))) for d in range(n)]
        table = rel[torch.tensor(row, device="cuda")]
        i = torch.arange(n, device="cuda")
        gap = (i[:, None] - i[None, :]).clamp(min=0)
        visible = (i[:, None] >= i[None, :]) & (i[:, None] // size == i[None, :] // size)
        o = _attend(_rms(q, eps), _rms(k, eps), v, x["scale"], visible, bias=lambda head: table[:, head][gap])
        return _mm(o.reshape(n, -1), W[p + "o"])
    left = _mix("left", design, h, W, p + "left.", x["left"], eps, kept, layer)
    r, q = x["right"], p + "right."
    H, D = r["heads"], r["dim"]
    out = []
    if kind == "parallel":
        before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        blend = lambda s: h + (before - h) * W[q + "mu." + s].to(F64)                                         # noqa: E731
        read, k, v = (_mm(blend(s), W[q + s]).view(n, H, D) for s in "rkv")
        w = torch.exp(-torch.exp(_mm(torch.tanh(_mm(blend("w"), W[q + "w1"])), W[q + "w2"]) + W[q + "w0"].to(F64))).view(n, H, D)
        u, S = W[q + "u"].to(F64)[:, :, None], torch.zeros((H, D, D), dtype=F64, device="cuda")
        for t in range(n):
            kv = k[t][:, :, None] * v[t][:, None, :]
            out.append(torch.bmm(read[t][:, None, :], S + u * kv)[:, 0])
            S = w[t][:, :, None] * S + kv
        o = _rms(torch.stack(out), eps).reshape(n, -1) * W[q + "norm"].to(F64) * _silu(_mm(blend("g"), W[q + "g"]))
        return x["left_scale"] * left + x["right_scale"] * _mm(o, W[q + "o"])
    rq, k, v = (_silu(_conv(_mm(h, W[q + s]), W[q + s + ".conv"])).view(n, -1, D) for s in "qkv")
    rq, k = (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (rq, k))
    rq, k = (y.repeat_interleave(H // y.shape[1], 1) for y in (rq * D ** -0.5, k))
    beta = torch.sigmoid(_mm(h, W[q + "b"]))[:, :, None]
    keep = torch.exp(-torch.exp(W[q + "A_log"].to(F64)) * torch.nn.functional.softplus(_mm(h, W[q + "a"]) + W[q + "dt_bias"].to(F64)))[:, :, None, None]
    S = torch.zeros((H, D, v.shape[2]), dtype=F64, device="cuda")
    for t in range(n):
        S = keep[t] * S
        u = beta[t] * (v[t] - torch.bmm(k[t][:, None, :], S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(torch.bmm(rq[t][:, None, :], S)[:, 0])
    o = (_rms(torch.stack(out), eps) * W[q + "norm"].to(F64)).reshape(n, -1) * _silu(_mm(h, W[q + "g"]))
    right = _mm(o, W[q + "o"])
    return 0.5 * (_rms(left, eps) * W[p + "left.out"].to(F64) + _rms(right, eps) * W[p + "right.out"].to(F64))


def _unit(design, h, W, p, mlp=None):
    if design == "Fasodra":
        return _mm(torch.relu(_mm(h, W[p + "up"])) ** 2, W[p + "down"])
    g, u = _mm(h, W[p + "gate"]), _mm(h, W[p + "up"])
    if design == "Vogilix":
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        return _mm(g * torch.sigmoid(1.702 * g) * (u + 1.0), W[p + "down"])
    return _mm(_silu(g) * u, W[p + "down"])


def _feed_forward(design, h, W, p, mlp):
    if mlp["kind"] == "dense":
        if design == "Zudepel":
            return _mm(_gelu_tanh(_mm(h, W[p + "gate"])) * _mm(h, W[p + "up"]), W[p + "down"])
        z = _mm(h, W[p + "up"])
        return _mm(0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0))), W[p + "down"])
    r = mlp["router"]
    z = _mm(h, W[p + "router"])
    if design == "Vogilix":
        value, chosen = z.topk(r["top"], 1)
        score = torch.sigmoid(value)
    else:
        s = torch.softmax(z, -1)
        c = s + W[p + "correction"].to(F64) if design == "Zudepel" else s
        if r.get("groups"):
            count, keep = r["groups"]["count"], r["groups"]["keep"]
            best = c.view(len(h), count, -1).max(-1).values.topk(keep, 1).indices
            kept = torch.zeros((len(h), count), dtype=torch.bool, device="cuda").scatter_(1, best, True)
            c = c.masked_fill(~kept.repeat_interleave(c.shape[1] // count, 1), -math.inf)
        chosen = c.topk(r["top"], 1).indices
        score = s.gather(1, chosen)
        score = score / (score.sum(-1, keepdim=True) + 1e-20)
    out = torch.zeros_like(h)
    for e in range(z.shape[1]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if not len(rows):
            continue
        weight = score[rows, place][:, None]
        if e >= r["experts"]:
            y = weight * h[rows]
        elif design == "Vogilix":
            y = _unit(design, weight * h[rows], W, "%se%d." % (p, e))
        else:
            y = weight * _unit(design, h[rows], W, "%se%d." % (p, e))
        out.index_add_(0, rows, y)
    if mlp.get("shared"):
        y = _unit(design, h, W, p + "shared.")
        out = out + (torch.sigmoid(_mm(h, W[p + "shared.sg"])) * y if design == "Zudepel" else y)
    return out


def _exact_design(cfg, W, sequences, wanted):
    design, eps, m = cfg["architecture"], cfg["norm"]["eps"], cfg.get("residual_mult", 1.0)
    out = []
    for tokens, wants in zip(sequences, wanted):
        ids, kept = torch.tensor(tokens, device="cuda"), {}
        x = W["embed"][ids].to(F64)
        if design == "Vogilix":
            x = x + W["pos"][:len(ids)].to(F64)
        w = lambda name: W[name].to(F64)                                                                      # noqa: E731

        def norm(name, v):
            if design == "Vogilix":
                return _rms(v, eps) * (1.0 + w(name))
            if design == "Fasodra":
                v = v - v.mean(-1, keepdim=True)
                return _rms(v, eps) * w(name) + w(name + ".b")
            return _rms(v, eps) * w(name)

        xs = [x, x]
        for i, layer in enumerate(cfg["layers"]):
            L, mlp = "l%d." % i, layer["mlp"]
            mix = lambda h: _mix(layer["type"], design, h, W, L + "mix.", layer["mixer"], eps, kept, i)       # noqa: E731
            ff = lambda h: _feed_forward(design, h, W, L + "mlp.", mlp)                                       # noqa: E731
            if design == "Vogilix":
                x = x + m * norm(L + "norm1", mix(x))
                x = x + m * norm(L + "norm2", ff(x))
                side = cfg["token_side"]["dim"]
                g = _gelu_tanh(_mm(x, W[L + "side.gate"])) * W["side.embed"][ids, i * side:(i + 1) * side].to(F64)
                x = x + m * _rms(_mm(g, W[L + "side.proj"]), eps) * w(L + "side.norm")
            elif design == "Zudepel":
                h = norm(L + "norm1", x)
                x = x + mix(h) + ff(h)
            else:
                for q, fn in (("1", mix), ("2", ff)):
                    a, b, c = w(L + "hc%s.in" % q), w(L + "hc%s.mix" % q), w(L + "hc%s.out" % q)
                    y = fn(norm(L + "norm" + q, a[0] * xs[0] + a[1] * xs[1]))
                    xs = [b[0, t] * xs[0] + b[1, t] * xs[1] + m * c[t] * y for t in range(2)]
        if design == "Fasodra":
            x = xs[0] + xs[1]
        out.append(_mm(norm("final.norm", x[wants]), W["head"]))
    return torch.stack(out)
