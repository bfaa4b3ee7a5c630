"""The work whose speed counts, as cases that a program times.

Two kinds of calls are here. Whole calls of the engine: a prompt (`Engine.prompt_step`) and a decode step
(`Engine.decode_step_device`, replayed as the generation loop replays it) of a Llama decoder whose logits come back. And
single sublayers, put together from the library's parts the way a layout names them: the norm in front, the mixer or the
routed feed-forward, and the norm behind it that adds its output to the residual stream; a prompt's sublayer is called
directly, a decode step's is captured once and replayed, as the engine does with the whole step. A sublayer returns the
residual stream, the normed stream and, where it has one, the per-sequence state it leaves.

Sizes are those of the repository's own benchmark (width 2,048 and 1,024, prompts of 2,048 tokens, decode steps of 1 to 64
sequences) or lie around them. Weights, streams and caches are drawn at random from the seed: matrices so that a product
keeps the size of its input, step sizes and decays over the ranges that such models are started with, cached keys, values
and latents of unit size.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from scriptling_llm_lib_b200 import models  # noqa: F401  (registers the architectures)
from scriptling_llm_lib_b200.config.llama import LlamaConfig
from scriptling_llm_lib_b200.engine import Engine, ModelLayout, StepContext, StepEntry, sequential_schedule
from scriptling_llm_lib_b200.models.llama import llama_layout
from scriptling_llm_lib_b200.parts.base import FEED_FORWARDS, PartSpec
from scriptling_llm_lib_b200.parts.block import LayerSpec
from scriptling_llm_lib_b200.parts.embedding import linear_head, token_embedding

DEVICE = "cuda:0"
PAGE = 64
VOCAB = 512          # of the sublayers' engines, whose embedding and head are not run
EPS = 1e-6
CONV = 4             # taps of the short convolutions
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# sizes by kind and width, as the repository's benchmark has them
SIZES = {
    "attention": {1024: dict(heads=8, kv=2, dim=64, vdim=128, window=512), 2048: dict(heads=16, kv=4, dim=64, vdim=128, window=1024)},
    "delta": {1024: dict(heads=8, kv=4, dim=128, vdim=128), 2048: dict(heads=16, kv=8, dim=128, vdim=128)},
    "rglru": {1024: dict(inner=1280, blocks=5), 2048: dict(inner=2560, blocks=10)},
    "latent": {1024: dict(heads=8, dim=128, rot=64, vdim=128, rank=256), 2048: dict(heads=16, dim=128, rot=64, vdim=128, rank=512)},
    "linear": {1024: dict(heads=8, dim=128, vdim=128), 2048: dict(heads=16, dim=128, vdim=128)},
    "scan": {1024: dict(inner=2048, state=16, rank=64), 2048: dict(inner=4096, state=16, rank=128)},
    "mamba2": {1024: dict(heads=32, dim=64, state=128, groups=1), 2048: dict(heads=64, dim=64, state=128, groups=1)},
    "experts": {1024: dict(experts=32, top=4, ff=704), 2048: dict(experts=64, top=6, ff=1408)},
}
LLAMA = {
    1024: dict(layers=4, heads=16, kv=4, head=64, ff=4096, vocab=8192),
    # the widths of the 1.7B decoder that the headline is quoted on, at a sixth of its depth and of its vocabulary
    2048: dict(layers=4, heads=32, kv=32, head=64, ff=8192, vocab=8192),
}


def _case(kind, phase, width, seqs, tokens=0, context=0, dtype="bfloat16", name=None):
    c = {"kind": kind, "phase": phase, "width": width, "seqs": seqs, "tokens": tokens, "context": context, "dtype": dtype}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one user waiting for the next token of a short answer: nothing but weights to read, launches and latency count
        _case("llama", "decode", 1024, 1, context=200, name="llama-decode-b1"),
        # the headline: eight users with long contexts, one token each
        _case("llama", "decode", 2048, 8, context=4096, name="llama-decode-b8"),
        # a prompt of the headline's length, the logits of its last token
        _case("llama", "prompt", 2048, 1, tokens=2048, name="llama-prompt"),
        # windowed attention whose values are wider than its keys: a prompt
        _case("attention", "prompt", 2048, 1, tokens=2048, name="attention-prompt"),
        # the gated delta rule: a prompt
        _case("delta", "prompt", 2048, 1, tokens=2048, name="delta-prompt"),
        # the gated linear recurrence in 32-bit, the precision of acceptance runs: several prompts of odd lengths in one step
        _case("rglru", "prompt", 1024, 3, tokens=1111, dtype="float32", name="rglru-prompt-f32"),
        # latent attention: a prompt, keys and values made per head
        _case("latent", "prompt", 2048, 1, tokens=2048, name="latent-prompt"),
        # latent attention: a decode step of eight users over the cached latents
        _case("latent", "decode", 2048, 8, context=4096, name="latent-decode-b8"),
        # linear attention with fixed decays: a prompt of an odd length
        _case("linear", "prompt", 2048, 1, tokens=3001, name="linear-prompt"),
        # the selective scan: a prompt
        _case("scan", "prompt", 2048, 1, tokens=2048, name="scan-prompt"),
        # the state-space recurrence with one decay a head: a decode step of a full batch
        _case("mamba2", "decode", 2048, 64, context=500, name="mamba2-decode-b64"),
        # routed experts behind a prompt
        _case("experts", "prompt", 2048, 1, tokens=2048, name="experts-prompt"),
    ]


def draw(rng):
    kind = rng.choice(["llama", "llama", *SIZES])
    width = rng.choice([1024, 2048])
    dtype = "float32" if rng.random() < 0.15 else "bfloat16"
    if rng.random() < 0.6:
        tokens = int(round(math.exp(rng.uniform(math.log(48), math.log(2048)))))
        seqs = rng.choice([1, 1, 2, 3, 5])
        if dtype == "float32":
            tokens = min(tokens, 300)
        return _case(kind, "prompt", width, seqs, tokens=max(tokens // seqs, 33), dtype=dtype)
    seqs = rng.choice([1, 2, 3, 4, 7, 8, 12, 16, 24, 32])
    context = int(round(math.exp(rng.uniform(math.log(20), math.log(4096 if seqs <= 8 else 2000)))))
    return _case(kind, "decode", width, seqs, context=context, dtype=dtype)


# --------------------------------------------------------------------------- what a case is made of
def _lengths(case):
    """Rows that every sequence brings: prompts of one step get shorter one after the other; one row in a decode step."""
    n = case["seqs"]
    if case["phase"] == "decode":
        return [1] * n
    return [max(1, case["tokens"] - i * case["tokens"] // (2 * n)) for i in range(n)]


def _contexts(case):
    """Positions that every sequence holds before the step: unequal ones in a batch of a decode step."""
    if case["phase"] == "prompt":
        return [0] * case["seqs"]
    return [case["context"] - (i * 37) % (case["context"] // 4 + 1) for i in range(case["seqs"])]


class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.g, device=DEVICE) * std + mean).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=self.g, device=DEVICE) * (hi - lo) + lo

    def ids(self, n, top):
        return torch.randint(0, top, (n,), generator=self.g, device=DEVICE, dtype=torch.int32)

    def step_bias(self, n):
        """Biases whose softplus is a step size between 0.001 and 0.1, evenly over its logarithm."""
        dt = torch.exp(self.uniform(n, lo=math.log(1e-3), hi=math.log(0.1)))
        return dt + torch.log(-torch.expm1(-dt))


def _weights(case, r):
    """The tensors of the sublayer by name, and the part that takes them."""
    kind, W, dt = case["kind"], case["width"], DTYPES[case["dtype"]]
    z = SIZES[kind][W]
    w = {}

    def matrix(name, rows, cols, std=None):
        w[name] = r.normal(rows, cols, std=std or cols ** -0.5, dtype=dt)

    def vector(name, n, mean=0.0, std=0.1):
        w[name] = r.normal(n, std=std, mean=mean, dtype=dt)

    vector("norm", W, mean=1.0)
    vector("post", W, mean=1.0)
    p = dict(hidden=W)
    if kind == "attention":
        H, G, D, V = z["heads"], z["kv"], z["dim"], z["vdim"]
        for n, rows in (("q", H * D), ("k", G * D), ("v", G * V)):
            matrix(n, rows, W)
        matrix("o", W, H * V)
        p.update(n_heads=H, n_kv_heads=G, head_dim=D, v_dim=V, window=z["window"], scale=D ** -0.5, value_norm_eps=EPS,
                 position=PartSpec("rotary", dict(head_dim=D, rotary_dim=D // 2, theta=10000.0, scaling=None, pairing="interleaved")),
                 q_name="q", k_name="k", v_name="v", o_name="o")
        return w, PartSpec("attention", p)
    if kind == "delta":
        H, G, D, V = z["heads"], z["kv"], z["dim"], z["vdim"]
        for n, rows in (("q", G * D), ("k", G * D), ("v", H * V), ("g", H * V)):
            matrix(n, rows, W)
        matrix("o", W, H * V)
        matrix("b", H, W)
        matrix("a", H, W, std=0.3 * W ** -0.5)
        for n, rows in (("q.conv", G * D), ("k.conv", G * D), ("v.conv", H * V)):
            w[n] = r.normal(rows, CONV, std=0.4, dtype=dt)
        w["A_log"] = torch.log(r.uniform(H, lo=1.0, hi=16.0)).to(dt)
        w["dt_bias"] = r.step_bias(H).to(dt)
        vector("onorm", V, mean=1.0)
        p.update(n_heads=H, n_kv_heads=G, key_dim=D, value_dim=V, conv_taps=CONV, norm_eps=EPS, q_name="q", k_name="k", v_name="v",
                 q_conv_name="q.conv", k_conv_name="k.conv", v_conv_name="v.conv", beta_name="b", decay_name="a", a_log_name="A_log",
                 dt_bias_name="dt_bias", gate_name="g", norm_name="onorm", o_name="o")
        return w, PartSpec("gated_delta_rule", p)
    if kind == "rglru":
        I, nb = z["inner"], z["blocks"]
        bs = I // nb
        matrix("y", I, W)
        matrix("x", I, W)
        matrix("o", W, I)
        for n in ("y.b", "x.b", "conv.b"):
            vector(n, I)
        w["conv"] = r.normal(I, CONV, std=0.4, dtype=dt)
        for n in ("ra", "ri"):
            w[n] = r.normal(nb, bs, bs, std=bs ** -0.5, dtype=dt)
            w[n + ".b"] = r.normal(nb, bs, std=0.1, dtype=dt)
        a = r.uniform(I, lo=0.9, hi=0.999)                          # the decay at a gate of one
        w["lam"] = torch.log(torch.expm1(-torch.log(a) / 8.0)).to(dt)
        p.update(width=I, blocks=nb, conv_taps=CONV, y_name="y", y_bias_name="y.b", x_name="x", x_bias_name="x.b", conv_name="conv",
                 conv_bias_name="conv.b", ra_name="ra", ra_bias_name="ra.b", ri_name="ri", ri_bias_name="ri.b", lam_name="lam", o_name="o")
        return w, PartSpec("rglru", p)
    if kind == "latent":
        H, D, P, V, R = z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
        matrix("q", H * (D + P), W)
        matrix("dkv", R + P, W)
        vector("dkv.norm", R, mean=1.0)
        matrix("uk", H * D, R)
        matrix("uv", H * V, R)
        matrix("o", W, H * V)
        p.update(n_heads=H, dim=D, rot_dim=P, v_dim=V, kv_rank=R, scale=(D + P) ** -0.5, norm_eps=EPS,
                 position=PartSpec("rotary", dict(head_dim=P, rotary_dim=P, theta=10000.0, scaling=None, pairing="interleaved")),
                 q_name="q", uk_name="uk", uv_name="uv", o_name="o", dkv_name="dkv", dkv_norm_name="dkv.norm")
        return w, PartSpec("latent_attention", p)
    if kind == "linear":
        H, D, V = z["heads"], z["dim"], z["vdim"]
        for n, rows in (("q", H * D), ("k", H * D), ("v", H * V), ("g", H * V)):
            matrix(n, rows, W)
        matrix("o", W, H * V)
        vector("onorm", H * V, mean=1.0)
        p.update(n_heads=H, key_dim=D, value_dim=V, decay=_decays(H), norm_eps=EPS, q_name="q", k_name="k", v_name="v", gate_name="g",
                 norm_name="onorm", o_name="o")
        return w, PartSpec("decay_linear_attention", p)
    if kind == "scan":
        I, N, K = z["inner"], z["state"], z["rank"]
        matrix("in", 2 * I, W)
        w["conv"] = r.normal(I, CONV, std=0.4, dtype=dt)
        vector("conv.b", I)
        matrix("x", K + 2 * N, I)
        matrix("dt", I, K, std=0.3 * K ** -0.5)
        w["dt.b"] = r.step_bias(I).to(dt)
        w["A_log"] = torch.log(torch.arange(1, N + 1, device=DEVICE, dtype=torch.float32)).expand(I, N).to(dt).contiguous()
        vector("D", I, mean=1.0)
        matrix("o", W, I)
        p.update(inner=I, n_state=N, dt_rank=K, conv_taps=CONV, in_name="in", conv_name="conv", conv_bias_name="conv.b", x_name="x",
                 dt_name="dt", dt_bias_name="dt.b", a_log_name="A_log", d_name="D", o_name="o")
        return w, PartSpec("selective_scan", p)
    if kind == "mamba2":
        H, V, N, G = z["heads"], z["dim"], z["state"], z["groups"]
        I = H * V
        matrix("in", 2 * I + 2 * G * N + H, W)
        w["conv"] = r.normal(I + 2 * G * N, CONV, std=0.4, dtype=dt)
        vector("conv.b", I + 2 * G * N)
        w["dt_bias"] = r.step_bias(H).to(dt)
        w["A_log"] = torch.log(r.uniform(H, lo=1.0, hi=16.0)).to(dt)
        vector("D", H, mean=1.0)
        vector("onorm", I, mean=1.0)
        matrix("o", W, I)
        p.update(n_heads=H, head_dim=V, n_state=N, n_groups=G, conv_taps=CONV, norm_groups=1, norm_eps=EPS, in_name="in", conv_name="conv",
                 conv_bias_name="conv.b", dt_bias_name="dt_bias", a_log_name="A_log", d_name="D", norm_name="onorm", o_name="o")
        return w, PartSpec("mamba2", p)
    E, F = z["experts"], z["ff"]
    matrix("router", E, W, std=3.0 * W ** -0.5)         # a trained router's logits are spread
    vector("router.b", E)
    names = {n: [f"e{j}.{n}" for j in range(E)] for n in ("gate", "up", "down")}
    for n, (rows, cols) in dict(gate=(F, W), up=(F, W), down=(W, F)).items():
        stack = r.normal(E, rows, cols, std=cols ** -0.5, dtype=dt)
        w.update(zip(names[n], stack))
    p.update(intermediate=F, experts=E, top=z["top"], n_groups=1, keep_groups=1, scale=1.0, router="top_softmax", router_name="router",
             correction_name="router.b", act="clamped_glu", gate_names=names["gate"], up_names=names["up"], down_names=names["down"],
             limit=7.0)
    return w, PartSpec("routed_experts", p)


def _decays(heads):
    return [1.0 - 2.0 ** (-5 - 3 * h / max(1, heads - 1)) for h in range(heads)]


def _state_shapes(case):
    """The per-sequence state that the sublayer keeps, by name."""
    kind = case["kind"]
    z = SIZES[kind][case["width"]]
    if kind == "delta":
        return {"S": (z["heads"], z["dim"], z["vdim"]), "conv": (CONV - 1, 2 * z["kv"] * z["dim"] + z["heads"] * z["vdim"])}
    if kind == "rglru":
        return {"S": (z["inner"],), "conv": (CONV - 1, z["inner"])}
    if kind == "linear":
        return {"S": (z["heads"], z["dim"], z["vdim"])}
    if kind == "scan":
        return {"S": (z["inner"], z["state"]), "conv": (CONV - 1, z["inner"])}
    if kind == "mamba2":
        return {"S": (z["heads"], z["state"], z["dim"]), "conv": (CONV - 1, z["heads"] * z["dim"] + 2 * z["groups"] * z["state"])}
    return {}


def _cached(case, r):
    """What every sequence's cache holds before a decode step: keys and values [positions, heads, width], or latents with
    their rotated key part (and no values)."""
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    if kind not in ("attention", "latent") or case["phase"] != "decode":
        return None
    z = SIZES[kind][case["width"]]
    heads, kw, vw = (z["kv"], z["dim"], z["vdim"]) if kind == "attention" else (1, z["rank"] + z["rot"], 0)
    return [(r.normal(n, heads, kw, dtype=dt), r.normal(n, heads, vw, dtype=dt) if vw else None) for n in _contexts(case)]


def _sublayer_inputs(case, seed):
    r = _Random(seed)
    w, part = _weights(case, r)
    rows = sum(_lengths(case))
    x = r.normal(rows, case["width"])
    state = {n: r.normal(case["seqs"], *shape, std=0.5) if case["phase"] == "decode" else None
             for n, shape in _state_shapes(case).items()}
    return w, part, x, state, _cached(case, r)


def _llama_inputs(case, seed):
    """Tensors by their checkpoint names, and the token ids of every sequence (its context, then the step's own)."""
    r, z, W, dt = _Random(seed), LLAMA[case["width"]], case["width"], DTYPES[case["dtype"]]
    raw = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": z["layers"], "hidden_size": W,
           "num_attention_heads": z["heads"], "num_key_value_heads": z["kv"], "head_dim": z["head"], "intermediate_size": z["ff"],
           "vocab_size": z["vocab"], "rope_theta": 10000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": False,
           "max_position_embeddings": 8192, "hidden_act": "silu"}
    w = {"model.embed_tokens.weight": r.normal(z["vocab"], W, dtype=dt), "lm_head.weight": r.normal(z["vocab"], W, std=W ** -0.5, dtype=dt),
         "model.norm.weight": r.normal(W, mean=1.0, std=0.1, dtype=dt)}
    for i in range(z["layers"]):
        p = f"model.layers.{i}."
        for n, rows, cols in (("self_attn.q_proj", z["heads"] * z["head"], W), ("self_attn.k_proj", z["kv"] * z["head"], W),
                              ("self_attn.v_proj", z["kv"] * z["head"], W), ("self_attn.o_proj", W, z["heads"] * z["head"]),
                              ("mlp.gate_proj", z["ff"], W), ("mlp.up_proj", z["ff"], W), ("mlp.down_proj", W, z["ff"])):
            w[p + n + ".weight"] = r.normal(rows, cols, std=cols ** -0.5, dtype=dt)
        for n in ("input_layernorm", "post_attention_layernorm"):
            w[p + n + ".weight"] = r.normal(W, mean=1.0, std=0.1, dtype=dt)
    ids = [r.ids(c + n, z["vocab"]) for c, n in zip(_contexts(case), _lengths(case))]
    return raw, w, ids


# --------------------------------------------------------------------------- preparing
def _pages(n):
    return -(-n // PAGE)


def prepare(case, seed):
    return _prepare_llama(case, seed) if case["kind"] == "llama" else _prepare_sublayer(case, seed)


def _prepare_llama(case, seed):
    raw, w, ids = _llama_inputs(case, seed)
    held = sum(_pages(len(i) + 1) for i in ids) * PAGE
    eng = Engine(llama_layout(LlamaConfig.from_dict(raw)), w, case["dtype"], held, case["seqs"], DEVICE)
    prompts = [i.tolist() for i in ids]
    if case["phase"] == "prompt":
        return {"engine": eng, "prompts": prompts}
    seqs = [eng.open() for _ in prompts]
    eng.prompt_step([StepEntry(s, p[:-1]) for s, p in zip(seqs, prompts)], 8192)
    return {"engine": eng, "seqs": seqs, "lengths": [s.length for s in seqs], "ids": torch.stack([i[-1] for i in ids])}


def _context(eng, seqs, lens, pos0):
    """A step's context for parts that are called by themselves, filled the way the engine fills it."""
    eng.cache.reserve([(s.slot, n) for s, n in zip(seqs, lens)])
    ctx = StepContext(eng)
    start = np.concatenate([[0], np.cumsum(lens)])
    tok_seq = np.repeat(np.arange(len(lens)), lens)
    arrays = dict(token_ids=np.zeros(start[-1]), tok_pos=np.arange(start[-1]) - start[tok_seq] + np.asarray(pos0)[tok_seq], tok_seq=tok_seq,
                  seq_start=start, seq_pos0=pos0, slots=[s.slot for s in seqs], want_rows=start[1:] - 1,
                  seq_pos_after=np.asarray(pos0) + np.asarray(lens))
    for name, a in arrays.items():
        setattr(ctx, name, torch.as_tensor(np.asarray(a, dtype=np.int32)).to(DEVICE))
    ctx.block_tables = [torch.as_tensor(np.ascontiguousarray(eng.cache.block_table(g, [s.slot for s in seqs]))).to(DEVICE)
                        for g in range(len(eng.cache.groups))]
    ctx.n_tokens, ctx.n_seqs, ctx.max_new = int(start[-1]), len(lens), max(lens)
    ctx.is_decode = max(lens) == 1
    ctx.seq_lens_host = None if ctx.is_decode else list(lens)
    ctx.from_start = not any(pos0)
    ctx.max_pages = max(_pages(p + n) for p, n in zip(pos0, lens))
    return ctx


def _prepare_sublayer(case, seed):
    w, part, x, state, cached = _sublayer_inputs(case, seed)
    W, lens, past = case["width"], _lengths(case), _contexts(case)
    rmsnorm = lambda name: PartSpec("rmsnorm", dict(width=W, eps=EPS, weight_name=name))        # noqa: E731
    mixer = part
    if part.kind == "routed_experts":       # the feed-forward is run by itself; its engine's layer has a small mixer
        w.update({n: torch.zeros((8, W) if n != "mo" else (W, 8), dtype=x.dtype, device=DEVICE) for n in ("mq", "mk", "mv", "mo")})
        mixer = PartSpec("attention", dict(hidden=W, n_heads=1, n_kv_heads=1, head_dim=8, position=None, q_name="mq", k_name="mk",
                                           v_name="mv", o_name="mo"))
    layout = ModelLayout(vocab_size=VOCAB, hidden_size=W, max_positions=8192, embedding=token_embedding(VOCAB, W, "embed"),
                         layers=(LayerSpec("pre_norm_input", {"mixer_norm": rmsnorm("norm"), "mixer": mixer}),),
                         schedule=sequential_schedule(1), final_norm=rmsnorm("post"), head=linear_head(VOCAB, W, "embed", tied=True))
    w["embed"] = torch.zeros((VOCAB, W), dtype=DTYPES[case["dtype"]], device=DEVICE)
    eng = Engine(layout, w, case["dtype"], sum(_pages(p + n) for p, n in zip(past, lens)) * PAGE, case["seqs"], DEVICE)
    block = eng.model.blocks[0]
    if part.kind == "routed_experts":
        ff = FEED_FORWARDS.build(part)
        ff.bind(w, DTYPES[case["dtype"]], torch.device(DEVICE))
        forward = lambda n, ctx: [ff.forward(n, ctx)]       # a list: float32 addends         # noqa: E731
    else:
        forward = lambda n, ctx: block.mixer.forward(n, ctx, 0, True)                           # noqa: E731
    seqs = [eng.open() for _ in lens]
    slots = torch.tensor([s.slot for s in seqs], device=DEVICE)
    kept = eng.cache.state.get(0) if state else None
    for n, v in state.items():
        if v is not None:
            kept[n][slots] = v
    if case["phase"] == "decode":
        eng.cache.reserve([(s.slot, p) for s, p in zip(seqs, past)])
        eng.cache.advance([(s.slot, p) for s, p in zip(seqs, past)])
    ctx = _context(eng, seqs, lens, past)
    if cached is not None:
        kpages, vpages = eng.cache.groups[0].unit_storage(0)
        for (keys, values), table in zip(cached, ctx.block_tables[0].long()):
            for pages, rows in ((kpages, keys), (vpages, values)):
                if rows is None:
                    continue
                full = torch.zeros((_pages(len(rows)) * PAGE, *rows.shape[1:]), dtype=rows.dtype, device=DEVICE)
                full[:len(rows)] = rows
                t = table[:_pages(len(rows))]
                seen = t >= 0                                       # pages behind a window are given back already
                pages[t[seen]] = full.view(-1, PAGE, *rows.shape[1:]).transpose(1, 2)[seen]

    def sublayer():
        residual = x.clone()
        y = forward(block.mixer_norm.forward(residual, None, ctx), ctx)
        normed = eng.model.final_norm.forward(residual, y, ctx)
        return (residual, normed, *(kept[n][:case["seqs"]] for n in state))

    s = {"engine": eng, "sublayer": sublayer}
    if case["phase"] == "decode":
        before = {n: kept[n].clone() for n in state}
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            sublayer()
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = sublayer()
        for n, v in before.items():
            kept[n].copy_(v)
    return s


# --------------------------------------------------------------------------- one pass
def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    if "sublayer" in state:
        return state["sublayer"]()
    eng = state["engine"]
    if "prompts" in state:
        seqs = [eng.open() for _ in state["prompts"]]
        logits, _ = eng.prompt_step([StepEntry(s, p) for s, p in zip(seqs, state["prompts"])])
        for s in seqs:
            s.close()
        return logits
    logits = eng.decode_step_device(state["seqs"], state["ids"])
    for s, n in zip(state["seqs"], state["lengths"]):       # the token is taken back, as a refused draft is
        eng.cache.length[s.slot] = n
    return logits


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    width = 2 if case["dtype"] == "bfloat16" else 4
    T, W = sum(_lengths(case)), case["width"]
    seen = sum(n * p + n * (n + 1) // 2 for n, p in zip(_lengths(case), _contexts(case)))       # (query, key) pairs
    held = sum(_contexts(case))
    if case["kind"] == "llama":
        z = LLAMA[W]
        layer = W * (2 * z["heads"] + 2 * z["kv"]) * z["head"] + 3 * W * z["ff"]
        rows = case["seqs"]                                                                     # of logits
        flops = 2 * T * layer * z["layers"] + 4 * seen * z["heads"] * z["head"] * z["layers"] + 2 * rows * W * z["vocab"]
        elements = z["layers"] * (layer + 2 * (held + T) * z["kv"] * z["head"]) + z["vocab"] * W + T * W
        return {"bytes": width * elements + 4 * rows * z["vocab"], "flops": flops}
    z, kind = SIZES[case["kind"]][W], case["kind"]
    state = 2 * case["seqs"] * sum(math.prod(s) for s in _state_shapes(case).values())          # read and written
    stream = T * W * (4 + 4 + width)                                                            # x, the residual stream, the normed one
    cache = 0
    if kind == "attention":
        weights = W * (z["heads"] * (z["dim"] + z["vdim"]) + z["kv"] * (z["dim"] + z["vdim"]))
        seen = sum(min(z["window"], p + i + 1) for n, p in zip(_lengths(case), _contexts(case)) for i in range(n))
        own = 2 * seen * z["heads"] * (z["dim"] + z["vdim"])
        cache = (sum(min(z["window"], p) for p in _contexts(case)) + T) * z["kv"] * (z["dim"] + z["vdim"])
    elif kind == "delta":
        weights = W * (2 * z["kv"] * z["dim"] + 3 * z["heads"] * z["vdim"] + 2 * z["heads"])
        own = 6 * T * z["heads"] * z["dim"] * z["vdim"]
    elif kind == "rglru":
        weights = 3 * W * z["inner"] + 2 * z["inner"] ** 2 // z["blocks"]
        own = 10 * T * z["inner"]
    elif kind == "latent":
        up = z["heads"] * (z["dim"] + z["vdim"]) * z["rank"]
        weights = W * (z["heads"] * (z["dim"] + z["rot"] + z["vdim"]) + z["rank"] + z["rot"]) + up
        if case["phase"] == "prompt":
            own = 2 * seen * z["heads"] * (z["dim"] + z["rot"] + z["vdim"])
        else:
            own = 2 * seen * z["heads"] * (2 * z["rank"] + z["rot"])
        cache = (held + T) * (z["rank"] + z["rot"])
    elif kind == "linear":
        weights = W * z["heads"] * (2 * z["dim"] + 3 * z["vdim"])
        own = 4 * T * z["heads"] * z["dim"] * z["vdim"]
    elif kind == "scan":
        weights = 3 * W * z["inner"] + z["inner"] * (2 * z["rank"] + 2 * z["state"])
        own = 6 * T * z["inner"] * z["state"]
    elif kind == "mamba2":
        inner = z["heads"] * z["dim"]
        weights = W * (3 * inner + 2 * z["groups"] * z["state"] + z["heads"])
        own = 6 * T * inner * z["state"]
    else:
        used = min(z["experts"], T * z["top"])
        weights = W * z["experts"] + 3 * used * W * z["ff"]
        own = 0
        return {"bytes": width * weights + stream, "flops": 2 * T * W * (z["experts"] + 3 * z["top"] * z["ff"])}
    return {"bytes": width * (weights + cache) + stream + 4 * state, "flops": 2 * T * weights + own}


def tolerance(case):
    """About four times what the two precisions are away from 64 bits: 3e-7 to 3e-6 and 0.002 to 0.004."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] in ("attention", "latent"):
        return {"rel": 8e-3, "max": 0.2}
    return {"rel": 1.5e-2, "max": 0.4}


# --------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    return _exact_llama(case, seed) if case["kind"] == "llama" else _exact_sublayer(case, seed)


def _rms(v, weight=1.0, eps=EPS):
    return v / torch.sqrt(v.square().mean(-1, keepdim=True) + eps) * weight


def _silu(v):
    return v * torch.sigmoid(v)


def _softplus(v):
    return torch.where(v > 0, v, torch.zeros_like(v)) + torch.log1p(torch.exp(-v.abs()))


def _turn(v, positions, dims, interleaved, theta=10000.0):
    """The leading `dims` of v [positions, heads, width] turned in neighbouring pairs or in halves."""
    freq = theta ** (-torch.arange(0, dims, 2, device=v.device, dtype=torch.float64) / dims)
    angle = positions.double()[:, None] * freq
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    out = v.clone()
    a, b = (v[..., 0:dims:2], v[..., 1:dims:2]) if interleaved else (v[..., :dims // 2], v[..., dims // 2:dims])
    ra, rb = a * c - b * s, a * s + b * c
    if interleaved:
        out[..., 0:dims:2], out[..., 1:dims:2] = ra, rb
    else:
        out[..., :dims // 2], out[..., dims // 2:dims] = ra, rb
    return out


def _attend(q, k, v, first, scale, window=0):
    """q [n, H, d] at positions from `first` on over k [m, G, d], v [m, G, e], position 0 first."""
    n, H = q.shape[:2]
    out = torch.empty((n, H, v.shape[-1]), dtype=q.dtype, device=q.device)
    at = torch.arange(n, device=q.device)[:, None] + first
    key = torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = key > at if not window else (key > at) | (key <= at - window)
    for h in range(H):
        g = h * k.shape[1] // H
        s = (q[:, h] @ k[:, g].T) * scale
        out[:, h] = s.masked_fill(hidden, -math.inf).softmax(-1) @ v[:, g]
    return out


def _exact_llama(case, seed):
    raw, w, ids = _llama_inputs(case, seed)
    w = {n: t.double() for n, t in w.items()}
    H, G, D = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"]
    rows = []
    for tokens in ids:
        x = w["model.embed_tokens.weight"][tokens.long()]
        n = x.shape[0]
        pos = torch.arange(n, device=x.device)
        for i in range(raw["num_hidden_layers"]):
            m = lambda name, v: v @ w[f"model.layers.{i}.{name}.weight"].T                        # noqa: E731
            h = _rms(x, w[f"model.layers.{i}.input_layernorm.weight"], 1e-5)
            q = _turn(m("self_attn.q_proj", h).view(n, H, D), pos, D, False)
            k = _turn(m("self_attn.k_proj", h).view(n, G, D), pos, D, False)
            v = m("self_attn.v_proj", h).view(n, G, D)
            x = x + m("self_attn.o_proj", _attend(q, k, v, 0, D ** -0.5).reshape(n, H * D))
            h = _rms(x, w[f"model.layers.{i}.post_attention_layernorm.weight"], 1e-5)
            x = x + m("mlp.down_proj", _silu(m("mlp.gate_proj", h)) * m("mlp.up_proj", h))
        rows.append(_rms(x[-1:], w["model.norm.weight"], 1e-5) @ w["lm_head.weight"].T)
    return torch.cat(rows)


def _convolve(v, filt, history, bias=0.0):
    """Behind `history`, the rows before v; and the rows that come to stand there after it."""
    rows = torch.cat([history, v])
    out = sum(rows[j:j + v.shape[0]] * filt[:, j] for j in range(CONV)) + bias
    return out, rows[-(CONV - 1):]


def _exact_sublayer(case, seed):
    w, part, x, state, cached = _sublayer_inputs(case, seed)
    w = {n: t.double() for n, t in w.items()}
    x = x.double()
    kind, z = case["kind"], SIZES[case["kind"]][case["width"]]
    shapes = _state_shapes(case)
    old = [{n: state[n][b].double() if state[n] is not None else torch.zeros(s, dtype=torch.float64, device=DEVICE)
            for n, s in shapes.items()} for b in range(case["seqs"])]
    h = _rms(x, w["norm"])
    ys, new, at = [], [], 0
    for b, (n, past) in enumerate(zip(_lengths(case), _contexts(case))):
        held = cached[b] if cached is not None else None
        y, after = _MIXERS[kind](h[at:at + n], w, z, old[b], held, past)
        ys.append(y)
        new.append(after)
        at += n
    out = x + torch.cat(ys)
    return (out, _rms(out, w["post"]), *(torch.stack([s[k] for s in new]) for k in shapes))


def _exact_attention(h, w, z, old, held, past):
    n, H, G, D, V = h.shape[0], z["heads"], z["kv"], z["dim"], z["vdim"]
    pos = torch.arange(past, past + n, device=h.device)
    q = _turn((h @ w["q"].T).view(n, H, D), pos, D // 2, True)
    k = _turn((h @ w["k"].T).view(n, G, D), pos, D // 2, True)
    v = _rms((h @ w["v"].T).view(n, G, V))
    if held is not None:
        k, v = torch.cat([held[0].double(), k]), torch.cat([held[1].double(), v])
    return _attend(q, k, v, past, D ** -0.5, z["window"]).reshape(n, H * V) @ w["o"].T, {}


def _exact_latent(h, w, z, old, held, past):
    n, H, D, P, V, R = h.shape[0], z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
    pos = torch.arange(past, past + n, device=h.device)
    q = (h @ w["q"].T).view(n, H, D + P)
    q = torch.cat([q[..., :D], _turn(q[..., D:], pos, P, True)], -1)
    down = h @ w["dkv"].T
    row = torch.cat([_rms(down[:, :R], w["dkv.norm"]), _turn(down[:, None, R:], pos, P, True)[:, 0]], -1)
    if held is not None:
        row = torch.cat([held[0][:, 0].double(), row])
    m = row.shape[0]
    k = torch.cat([(row[:, :R] @ w["uk"].T).view(m, H, D), row[:, None, R:].expand(m, H, P)], -1)
    v = (row[:, :R] @ w["uv"].T).view(m, H, V)
    return _attend(q, k, v, past, (D + P) ** -0.5).reshape(n, H * V) @ w["o"].T, {}


def _exact_delta(h, w, z, old, held, past):
    n, H, G, D, V = h.shape[0], z["heads"], z["kv"], z["dim"], z["vdim"]
    raw = torch.cat([h @ w["q"].T, h @ w["k"].T, h @ w["v"].T], -1)
    c, conv = _convolve(raw, torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]]), old["conv"])
    q, k, v = _silu(c).split([G * D, G * D, H * V], -1)
    unit = lambda t: t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)                     # noqa: E731
    q = (unit(q.view(n, G, D)) * D ** -0.5).repeat_interleave(H // G, 1)
    k = unit(k.view(n, G, D)).repeat_interleave(H // G, 1)
    v = v.view(n, H, V)
    beta = torch.sigmoid(h @ w["b"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * _softplus(h @ w["a"].T + w["dt_bias"]))
    S, rows = old["S"].clone(), []
    for t in range(n):
        S = S * decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None]
        rows.append(torch.einsum("hdv,hd->hv", S, q[t]))
    o = _rms(torch.stack(rows), w["onorm"]) * _silu((h @ w["g"].T).view(n, H, V))
    return o.reshape(n, H * V) @ w["o"].T, {"S": S, "conv": conv}


def _exact_rglru(h, w, z, old, held, past):
    n, I, nb = h.shape[0], z["inner"], z["blocks"]
    y = h @ w["y"].T + w["y.b"]
    y = 0.5 * y * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (y + 0.044715 * y ** 3)))
    u, conv = _convolve(h @ w["x"].T + w["x.b"], w["conv"], old["conv"], w["conv.b"])
    ub = u.view(n, nb, I // nb)
    r, i = (torch.sigmoid(torch.einsum("nbk,bjk->nbj", ub, w[g]) + w[g + ".b"]).reshape(n, I) for g in ("ra", "ri"))
    log_a = -8.0 * r * _softplus(w["lam"])
    a, b = log_a.exp(), torch.sqrt(-torch.expm1(2.0 * log_a)) * i * u
    S, rows = old["S"].clone(), []
    for t in range(n):
        S = a[t] * S + b[t]
        rows.append(S)
    return (torch.stack(rows) * y) @ w["o"].T, {"S": S, "conv": conv}


def _exact_linear(h, w, z, old, held, past):
    n, H, D, V = h.shape[0], z["heads"], z["dim"], z["vdim"]
    q, k, v = (_silu(h @ w[m].T).view(n, H, -1) for m in ("q", "k", "v"))
    g = torch.tensor(_decays(H), dtype=torch.float32).double().to(h.device)[:, None, None]
    S, rows = old["S"].clone(), []
    for t in range(n):
        S = g * S + k[t, :, :, None] * v[t, :, None]
        rows.append(torch.einsum("hdv,hd->hv", S, q[t]))
    o = _rms(torch.stack(rows).reshape(n, H * V), w["onorm"]) * torch.sigmoid(h @ w["g"].T)
    return o @ w["o"].T, {"S": S}


def _exact_scan(h, w, z, old, held, past):
    n, I, N, K = h.shape[0], z["inner"], z["state"], z["rank"]
    raw, gate = (h @ w["in"].T).split(I, -1)
    c, conv = _convolve(raw, w["conv"], old["conv"], w["conv.b"])
    c = _silu(c)
    low, B, C = (c @ w["x"].T).split([K, N, N], -1)
    dt = _softplus(low @ w["dt"].T + w["dt.b"])
    A = -torch.exp(w["A_log"])
    S, rows = old["S"].clone(), []
    for t in range(n):
        S = torch.exp(dt[t, :, None] * A) * S + (dt[t] * c[t])[:, None] * B[t]
        rows.append(S @ C[t])
    return ((torch.stack(rows) + w["D"] * c) * _silu(gate)) @ w["o"].T, {"S": S, "conv": conv}


def _exact_mamba2(h, w, z, old, held, past):
    n, H, V, N, G = h.shape[0], z["heads"], z["dim"], z["state"], z["groups"]
    I = H * V
    gate, raw, dt = (h @ w["in"].T).split([I, I + 2 * G * N, H], -1)
    c, conv = _convolve(raw, w["conv"], old["conv"], w["conv.b"])
    c, B, C = _silu(c).split([I, G * N, G * N], -1)
    c = c.reshape(n, H, V)
    B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    dt = _softplus(dt + w["dt_bias"])
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)
    S, rows = old["S"].clone(), []
    for t in range(n):
        S = decay[t, :, None, None] * S + (dt[t, :, None] * B[t])[:, :, None] * c[t, :, None]
        rows.append(torch.einsum("hnv,hn->hv", S, C[t]))
    y = (torch.stack(rows) + w["D"][:, None] * c).reshape(n, I) * _silu(gate)
    return _rms(y, w["onorm"]) @ w["o"].T, {"S": S, "conv": conv}


def _exact_experts(h, w, z, old, held, past):
    top, picked = (h @ w["router"].T + w["router.b"]).topk(z["top"], -1)
    share = top.softmax(-1)
    y = torch.zeros_like(h)
    for j in range(z["experts"]):
        row, place = (picked == j).nonzero(as_tuple=True)
        g = (h[row] @ w[f"e{j}.gate"].T).clamp(max=7.0)
        u = (h[row] @ w[f"e{j}.up"].T).clamp(-7.0, 7.0)
        y[row] += ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[f"e{j}.down"].T) * share[row, place, None]
    return y, {}


_MIXERS = {"attention": _exact_attention, "latent": _exact_latent, "delta": _exact_delta, "rglru": _exact_rglru, "linear": _exact_linear,
           "scan": _exact_scan, "mamba2": _exact_mamba2, "experts": _exact_experts}
