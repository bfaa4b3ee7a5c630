"""The Muvorax decoder on the GPU against the plain statement in plain_muvorax.py: each mechanism
alone, the residual stream layer by layer, whole prompts against token-by-token decoding and
against portions, unequal batches, slots and pages used again, far keys and page borders, the first
tokens, long decoding, other sizes, greedy generation through the entry point. Configurations and
weights are made here; weights are larger than a trained model's so that every branch moves the
logits."""
import json
import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import plain_muvorax as plain
from scriptling_llm_lib_b200.csrc.bindings import KernelSet

pytestmark = pytest.mark.gpu

TOL_F32 = 2e-4       # of a row's largest logit
TOL_BF16 = 6e-2
YARN = {"factor": 4.0, "fast": 16.0, "original": 64, "slow": 2.0}


def latent(heads=3, dim=8, rot_dim=4, vdim=12, rank=20, scale=0.4, base=100.0, dims=None, scaling=None, kv_from=None):
    rot = {"base": base, "dims": rot_dim if dims is None else dims}
    if scaling is not None:
        rot["scaling"] = scaling
    m = {"dim": dim, "heads": heads, "kv_rank": rank, "rot": rot, "rot_dim": rot_dim, "scale": scale, "vdim": vdim}
    if kv_from is not None:
        m["kv_from"] = kv_from
    return {"type": "latent_attention", "mixer": m}


def lightning(heads=3, dim=8, vdim=12, decay=(0.5, 0.9, 0.99)):
    return {"type": "lightning", "mixer": {"decay": list(decay), "dim": dim, "heads": heads, "vdim": vdim}}


def mamba(inner=40, state=6, dt_rank=5, conv=3):
    return {"type": "mamba1", "mixer": {"conv": conv, "dt_rank": dt_rank, "inner": inner, "state": state}}


def dense(ff):
    return {"ff": ff, "kind": "dense"}


def moe(ff=24, experts=8, top=2, count=2, keep=1, scale=1.5):
    return {"expert": {"ff": ff}, "kind": "moe", "router": {"experts": experts, "groups": {"count": count, "keep": keep}, "scale": scale,
                                                            "top": top}}


def with_ff(layer, mlp):
    return dict(layer, mlp=mlp)


def config(layers, width=64, vocab=96, eps=1e-6):
    return {"architecture": "Muvorax", "layers": [dict({"mlp": None}, **l) for l in layers], "norm": {"eps": eps}, "vocab": vocab,
            "width": width}


# Sizes that differ from one another in every number. A: every kind of layer once or twice, a layer
# reading another's latent with other head counts, a layer without a feed-forward. B: ten heads (two
# groups of the attention kernel's warps), a latent that is no multiple of 32, value columns that are
# no multiple of 4, one tap, a rotation of fewer dims than the rotated part and without rescaling,
# nine experts in three groups of which two are kept. C: one group of experts, one expert a token,
# decays of exactly 0 and 1, many states per channel.
CFG_A = config([with_ff(lightning(), moe()), with_ff(latent(scaling=YARN), dense(80)), with_ff(mamba(), moe(16, 6, 3, 3, 2, 0.7)),
                latent(5, 6, 4, 10, 20, 0.3, scaling=YARN, kv_from=1), with_ff(lightning(2, 16, 4, (0.2, 0.999)), dense(40))])
CFG_B = config([with_ff(latent(10, 12, 8, 6, 72, 0.25, 5000.0, dims=6), moe(40, 9, 3, 3, 2, 2.5)), mamba(56, 17, 3, 1),
                with_ff(lightning(2, 40, 50, (0.97, 0.6)), dense(72)), with_ff(latent(4, 16, 8, 20, 72, 0.2, 5000.0, dims=6, kv_from=0),
                                                                               moe(8, 4, 1, 1, 1, 1.0))],
               width=96, vocab=130, eps=1e-5)
CFG_C = config([with_ff(mamba(24, 40, 8, 4), moe(12, 5, 1, 1, 1, 3.0)), with_ff(lightning(4, 4, 24, (0.0, 1.0, 0.8, 0.95)), moe(20, 4, 4, 2, 2, 1.0)),
                with_ff(latent(1, 20, 2, 32, 130, 0.5, 20.0), dense(24))], width=40, vocab=77)


# widths that are multiples of nothing: every vector path has to step aside
CFG_D = config([with_ff(latent(3, 5, 2, 3, 9, 0.6, 30.0), moe(6, 3, 2, 1, 1, 1.2)), with_ff(mamba(10, 1, 1, 2), dense(14)),
                with_ff(lightning(1, 5, 7, (0.9,)), moe(10, 6, 1, 3, 1, 0.5)), latent(1, 3, 2, 5, 9, 0.4, 30.0, kv_from=0),
                mamba(6, 3, 2, 5)], width=50, vocab=61)


def random_weights(cfg, seed, std=0.25):
    """Weights by tensor name for `cfg`, bfloat16-representable (the folder stores bfloat16)."""
    from scriptling_llm_lib_b200 import models  # noqa: F401
    from scriptling_llm_lib_b200.config.registry import architecture_for
    from scriptling_llm_lib_b200.engine.model import DecoderModel
    arch = architecture_for("Muvorax")
    specs = DecoderModel(arch.layout(arch.config_class.from_dict(cfg, "test"))).tensor_specs()
    g = torch.Generator().manual_seed(seed)
    W = {}
    for s in specs:
        t = torch.randn(s.shape, generator=g)
        if s.init == "norm_weight":
            t = 1.0 + 0.2 * t
        elif s.init == "slope":
            t = 0.8 + 0.1 * t
        elif s.init == "matrix":
            t = t * std * (4.0 / math.sqrt(s.shape[-1]))
        elif s.init == "bias":
            t = 0.3 * t
        else:
            t = 0.5 * t
        W[s.name] = t.to(torch.bfloat16)
    W["embed"] = torch.randn(W["embed"].shape, generator=g).to(torch.bfloat16)
    return W


def write_folder(path, cfg, W):
    from scriptling_llm_lib_b200.weights.safetensors_io import write_safetensors
    path.mkdir(parents=True, exist_ok=True)
    (path / "config.json").write_text(json.dumps(cfg))
    write_safetensors(path / "model.safetensors", W)
    return path


def ids(n, vocab, seed):
    return [int(t) for t in np.random.default_rng(seed).integers(0, vocab, n)]


def engine(folder, dtype="float32", max_tokens=2048, max_seqs=8, **kw):
    from scriptling_llm_lib_b200.engine.step import Engine
    return Engine.from_folder(folder, dtype, max_tokens=max_tokens, max_seqs=max_seqs, **kw)


def run(eng, pieces):
    """Feed one sequence in the given pieces; logits of every position [T, vocab]."""
    from scriptling_llm_lib_b200.engine.step import StepEntry
    seq = eng.open()
    out = []
    for p in pieces:
        out.append(eng.step([StepEntry(seq, list(p), list(range(len(p))))]))
    eng.check_errors()
    seq.close()
    return torch.cat(out).cpu().double()


def cut(tokens, sizes):
    out, at = [], 0
    for s in sizes:
        out.append(tokens[at:at + s])
        at += s
    if at < len(tokens):
        out.append(tokens[at:])
    return [p for p in out if p]


def rel(got, want):
    return float(((got - want).abs().amax(-1) / want.abs().amax(-1).clamp_min(1e-30)).max())


@pytest.fixture(scope="module")
def folders(tmp_path_factory):
    root = tmp_path_factory.mktemp("muvorax")
    out = {}
    for name, cfg, seed in (("A", CFG_A, 1), ("B", CFG_B, 2), ("C", CFG_C, 3), ("D", CFG_D, 4)):
        W = random_weights(cfg, seed)
        out[name] = (write_folder(root / name, cfg, W), cfg, W)
    return out


def plain_logits(cfg, W, tokens, rnd=plain.ident, layers_out=None):
    return plain.PlainMuvorax(cfg, W, rnd).forward(tokens, layers_out)


# --------------------------------------------------------------------------- whole models
@pytest.mark.parametrize("name", ["A", "B", "C", "D"])
def test_a_whole_prompt_equals_the_plain_statement_in_32_bit(folders, name):
    folder, cfg, W = folders[name]
    tokens = ids(90, cfg["vocab"], 10)
    want = plain_logits(cfg, W, tokens)
    got = run(engine(folder), [tokens])
    assert rel(got, want) < TOL_F32


@pytest.mark.parametrize("name", ["A", "B", "C", "D"])
def test_bfloat16_stays_near_the_plain_statement_that_rounds_where_the_engine_stores(folders, name):
    folder, cfg, W = folders[name]
    tokens = ids(70, cfg["vocab"], 11)
    want = plain_logits(cfg, W, tokens)
    want16 = plain_logits(cfg, W, tokens, rnd=plain.bf16_round)
    eng = engine(folder, "bfloat16")
    got = run(eng, [tokens])
    assert rel(got, want16) < TOL_BF16 and rel(got, want) < 2 * TOL_BF16
    step = run(eng, [tokens[:50]] + [[t] for t in tokens[50:]])
    assert rel(step, got) < TOL_BF16


def test_the_residual_stream_after_every_layer(folders):
    from scriptling_llm_lib_b200.engine.step import StepEntry
    folder, cfg, W = folders["A"]
    tokens = ids(37, cfg["vocab"], 12)
    want = []
    plain_logits(cfg, W, tokens, layers_out=want)
    eng = engine(folder)
    seq = eng.open()
    arr = np.asarray(tokens, dtype=np.int64)
    eng.cache.reserve([(seq.slot, len(tokens))])
    ctx = eng._context([StepEntry(seq, tokens, [])], arr, [len(tokens)], [0], [])
    x = eng.model.embedding.forward(ctx.token_ids, ctx)
    delta = None
    for i, e in enumerate(eng.layout.schedule):
        delta = eng.model.blocks[e.layer].forward(x, delta, ctx, e.cache_unit, e.writes_cache)
        y = delta.y.double()
        y = y.sum(0) if y.dim() == 3 else y
        w, b, a = delta.norm.terms()
        full = x.double() + torch.tanh(a * y) * w.double() + b.double()
        assert float((full.cpu() - want[i]).abs().max()) < 1e-4 * float(want[i].abs().max()), f"layer {i}"
    seq.close()


@pytest.mark.parametrize("layer", [lightning(), latent(scaling=YARN), mamba(), with_ff(lightning(1, 4, 4, (0.9,)), moe()),
                                   with_ff(mamba(8, 2, 1, 2), dense(48)), latent(2, 4, 0, 8, 6, 1.0, dims=0), mamba(20, 12, 4, 3),
                                   mamba(12, 70, 2, 2)],
                         ids=["lightning", "latent", "scan", "experts", "dense", "latent-without-rotation", "scan-12-states", "scan-70-states"])
def test_each_mechanism_alone(tmp_path, layer):
    cfg = config([layer], width=32, vocab=50)
    W = random_weights(cfg, 5, std=0.4)
    folder = write_folder(tmp_path / "m", cfg, W)
    tokens = ids(45, 50, 13)
    want = plain_logits(cfg, W, tokens)
    eng = engine(folder)
    assert rel(run(eng, [tokens]), want) < TOL_F32
    assert rel(run(eng, [tokens[:20]] + [[t] for t in tokens[20:]]), want) < TOL_F32


@pytest.mark.parametrize("rank,heads,dtype", [(160, 2, "float32"), (264, 9, "float32"), (512, 3, "float32"), (256, 4, "bfloat16")])
def test_wide_latents_token_by_token(tmp_path, rank, heads, dtype):
    """Latents of several hundred: every lane of the attention kernel owns several groups of columns."""
    cfg = config([latent(heads, 8, 8, 8, rank, 0.5, 1000.0), with_ff(latent(2, 4, 8, 12, rank, 0.3, 1000.0, kv_from=0), dense(16))],
                 width=32, vocab=40)
    W = random_weights(cfg, 9, std=0.4)
    folder = write_folder(tmp_path / "m", cfg, W)
    tokens = ids(75, 40, 21)
    eng = engine(folder, dtype)
    got = run(eng, [tokens[:3]] + [[t] for t in tokens[3:]])
    if dtype == "float32":
        assert rel(got, plain_logits(cfg, W, tokens)) < TOL_F32
    else:
        assert rel(got, plain_logits(cfg, W, tokens, rnd=plain.bf16_round)) < TOL_BF16


# --------------------------------------------------------------------------- cutting, batches, slots
@pytest.mark.parametrize("name", ["A", "B", "C", "D"])
def test_token_by_token_and_portions_equal_the_whole_prompt(folders, name):
    folder, cfg, W = folders[name]
    tokens = ids(150, cfg["vocab"], 14)
    want = plain_logits(cfg, W, tokens)
    eng = engine(folder)
    for sizes in ([1] * 150, [2] * 75, [3, 2, 31, 33, 1, 64], [64, 64], [63, 2, 63], [100] + [1] * 50):
        got = run(eng, cut(tokens, sizes))
        assert rel(got, want) < TOL_F32, sizes


def test_unequal_requests_in_a_batch_equal_each_alone_and_slots_are_used_again(folders):
    from scriptling_llm_lib_b200.engine.step import StepEntry
    folder, cfg, W = folders["B"]
    V = cfg["vocab"]
    reqs = [ids(n, V, 20 + i) for i, n in enumerate((70, 3, 129, 1, 40))]
    prompt = [60, 2, 100, 1, 33]
    want = [plain_logits(cfg, W, r) for r in reqs]
    eng = engine(folder, max_seqs=6)
    for round_ in range(3):                     # the same slots and pages again, after other requests held them
        seqs = [eng.open() for _ in reqs]
        out = eng.step([StepEntry(s, r[:p], list(range(p))) for s, r, p in zip(seqs, reqs, prompt)]).cpu().double()
        got, at = [[] for _ in reqs], 0
        for i, p in enumerate(prompt):
            got[i].append(out[at:at + p])
            at += p
        pos = list(prompt)
        live = [i for i in range(len(reqs)) if pos[i] < len(reqs[i])]
        for i in range(len(reqs)):
            if i not in live:
                seqs[i].close()
        while live:
            out = eng.step([StepEntry(seqs[i], [reqs[i][pos[i]]], [0]) for i in live]).cpu().double()
            for j, i in enumerate(live):
                got[i].append(out[j:j + 1])
                pos[i] += 1
                if pos[i] == len(reqs[i]):
                    seqs[i].close()
            live = [i for i in live if pos[i] < len(reqs[i])]
        for i in range(len(reqs)):
            assert rel(torch.cat(got[i]), want[i]) < TOL_F32, (round_, i)
        reqs, prompt, want = reqs[::-1], prompt[::-1], want[::-1]
    assert eng.cache.slots.n_held == 0 and all(g.pool.n_held == 0 for g in eng.cache.groups)


def test_the_first_tokens_of_a_sequence(folders):
    folder, cfg, W = folders["A"]
    eng = engine(folder)
    for n in (1, 2, 3, 4):
        tokens = ids(n, cfg["vocab"], 30 + n)
        want = plain_logits(cfg, W, tokens)
        assert rel(run(eng, [tokens]), want) < TOL_F32
        assert rel(run(eng, [[t] for t in tokens]), want) < TOL_F32


def test_long_decoding_keeps_the_states(folders):
    folder, cfg, W = folders["C"]
    tokens = ids(260, cfg["vocab"], 15)
    want = plain_logits(cfg, W, tokens)
    got = run(engine(folder), [tokens[:5]] + [[t] for t in tokens[5:]])
    assert rel(got, want) < TOL_F32


# --------------------------------------------------------------------------- far keys and page borders
def test_one_loud_key_far_back_and_at_page_borders(tmp_path):
    """One key that carries every later row. A token of its own (the last id) lights channel 0 of the
    stream, the down-projection turns that into the latent's first component, head 0's first key dim
    reads it, and every query has a constant there: so wherever that token stands, at the first
    position, far back, or on either side of a page border, the rows behind it take their output from
    its cached latent; in a prompt and token by token."""
    cfg = config([with_ff(latent(2, 8, 4, 8, 12, 2.0, 50.0), dense(32))], width=32, vocab=40)
    W = random_weights(cfg, 7, std=0.5)
    loud = 39
    W["embed"][:, 0] = 0.0
    W["embed"][loud, 0] = 8.0
    for name, v0, v1 in (("l0.norm1", 1.0, 0.0), ("l0.norm1.b", 0.0, 1.0)):       # channel 0 passes, channel 1 is the constant 1
        W[name][0], W[name][1] = v0, v1
    W["l0.mix.dkv"][0, :] = 0.0
    W["l0.mix.dkv"][0, 0] = 10.0
    W["l0.mix.dkv.norm"][0] = 1.0
    W["l0.mix.uk"][0, :] = 0.0
    W["l0.mix.uk"][0, 0] = 1.0
    W["l0.mix.q"][0, :] = 0.0
    W["l0.mix.q"][0, 1] = 5.0
    folder = write_folder(tmp_path / "m", cfg, W)
    eng = engine(folder)
    base = ids(200, 39, 16)                          # never the loud token
    other = plain_logits(cfg, W, base)
    for p in (0, 1, 63, 64, 65, 127, 128, 150):
        tokens = list(base)
        tokens[p] = loud
        want = plain_logits(cfg, W, tokens)
        assert rel(want[190:], other[190:]) > 100 * TOL_F32         # the far key shows in the last rows
        assert rel(run(eng, [tokens]), want) < TOL_F32
        assert rel(run(eng, [tokens[:170]] + [[t] for t in tokens[170:]]), want) < TOL_F32


def test_a_slowly_decaying_head_remembers_the_first_token(tmp_path):
    cfg = config([lightning(2, 8, 8, (1.0, 0.5))], width=24, vocab=30)
    W = random_weights(cfg, 8, std=0.5)
    folder = write_folder(tmp_path / "m", cfg, W)
    eng = engine(folder)
    a = ids(140, 30, 17)
    b = [(a[0] + 3) % 30] + a[1:]
    wa, wb = plain_logits(cfg, W, a), plain_logits(cfg, W, b)
    assert rel(wa[130:], wb[130:]) > 10 * TOL_F32
    for tokens, want in ((a, wa), (b, wb)):
        assert rel(run(eng, [tokens]), want) < TOL_F32
        assert rel(run(eng, [tokens[:33]] + [[t] for t in tokens[33:]]), want) < TOL_F32


# --------------------------------------------------------------------------- kernels by themselves
def test_the_router_against_the_plain_choice():
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k = KernelSet(torch.float32).mix
    g = torch.Generator().manual_seed(3)
    for E, groups, keep, top in ((8, 2, 1, 2), (12, 4, 2, 3), (6, 1, 1, 6), (9, 9, 3, 3), (64, 8, 3, 6), (5, 5, 5, 1)):
        h = torch.randn(50, 24, generator=g)
        wr = torch.randn(E, 24, generator=g)
        corr = torch.randn(E, generator=g) * 1.5          # corrections large enough to make choice scores negative
        Wd = {"r.router": wr.double(), "r.correction": corr.double()}
        want_idx, want_w = plain.route(h.double(), Wd, "r.", {"experts": E, "top": top, "scale": 1.7, "groups": {"count": groups, "keep": keep}})
        idx = torch.empty((50, top), dtype=torch.int32, device="cuda")
        wgt = torch.empty((50, top), dtype=torch.float32, device="cuda")
        k.moe_route((h @ wr.T).cuda().contiguous(), corr.cuda(), idx, wgt, groups, keep, top, 1.7)
        for t in range(50):
            got = dict(zip(idx[t].tolist(), wgt[t].tolist()))
            want = dict(zip(want_idx[t].tolist(), want_w[t].tolist()))
            assert set(got) == set(want), (E, t)
            assert all(abs(got[e] - want[e]) < 1e-5 for e in want)


def test_linear_attention_in_pieces_against_the_recurrence():
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k = KernelSet(torch.float32).mix
    g = torch.Generator().manual_seed(4)
    H, D, V = 3, 10, 22
    lens = [1, 31, 32, 33, 70, 4]
    T = sum(lens)
    proj = torch.randn(T, 2 * H * D + H * V + 5, generator=g)
    decay = torch.tensor([0.3, 0.95, 1.0])
    start = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    state0 = torch.randn(len(lens) + 2, H, D, V, generator=g) * 0.3
    ctx = SimpleNamespace(seq_start=torch.from_numpy(start).cuda(), slots=torch.tensor([5, 0, 3, 1, 6, 2], dtype=torch.int32).cuda(),
                          n_seqs=len(lens), max_new=max(lens), engine=SimpleNamespace(sm_count=148))
    st = state0.clone().cuda()
    o = torch.empty((T, H * V), dtype=torch.float32, device="cuda")
    k.lin_attn_decay(proj.cuda(), 0, H * D, 2 * H * D, decay.cuda(), st, ctx, o, H, D, V)
    p = proj.double()
    q = plain.silu(p[:, :H * D]).view(T, H, D)
    kk = plain.silu(p[:, H * D:2 * H * D]).view(T, H, D)
    v = plain.silu(p[:, 2 * H * D:2 * H * D + H * V]).view(T, H, V)
    for b, slot in enumerate([5, 0, 3, 1, 6, 2]):
        for h in range(H):
            S = state0[slot, h].double()
            for t in range(start[b], start[b + 1]):
                S = float(decay[h]) * S + torch.outer(kk[t, h], v[t, h])
                want = S.T @ q[t, h]
                assert float((o[t].cpu().double().view(H, V)[h] - want).abs().max()) < 1e-4 * max(1.0, float(want.abs().max()))
            assert float((st[slot, h].cpu().double() - S).abs().max()) < 1e-4 * max(1.0, float(S.abs().max()))
    assert torch.equal(st[4].cpu(), state0[4])          # a slot no sequence of the step holds is left alone


@pytest.mark.parametrize("H, D, P, V, R", [(16, 128, 64, 128, 512), (5, 40, 8, 24, 72), (20, 64, 0, 40, 256), (33, 8, 24, 8, 328), (4, 256, 16, 200, 120)])
@pytest.mark.parametrize("window, n_split", [(0, 1), (0, 5), (100, 3)])
def test_latent_decode_on_the_tensor_cores(H, D, P, V, R, window, n_split):
    """The absorbed queries, scores and sums over the latent, merge and values against the formula, kernel by kernel on what the one
    before left: one position to several pages, pages scattered, unused rows NaN, heads that leave a block partly empty, splits that
    get no key, sink and gates. Float sums of products exact in their parts: 2e-6 sqrt(width) of the largest element; values rounded
    to 8 bits."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k = KernelSet(torch.bfloat16).mix
    assert k.latent.takes(D, P, V, R) and not k.latent.takes(D, P, V, 520) and not k.latent.takes(D + 4, P, V, R)
    g = torch.Generator().manual_seed(R + H)
    lens = [1, 64, 65, 200, 333, 130]
    B, W = len(lens), R + P
    need = [-(-n // 64) for n in lens]
    table = torch.zeros(B, max(need), dtype=torch.int32)
    order = torch.randperm(sum(need) + 2, generator=g).tolist()
    pages = torch.full((sum(need) + 2, 1, 64, W), float("nan"))
    rows = [torch.randn(n, W, generator=g).bfloat16() for n in lens]
    for b, n in enumerate(lens):
        for i in range(need[b]):
            table[b, i] = order.pop()
            part = rows[b][64 * i:64 * (i + 1)]
            pages[table[b, i], 0, :len(part)] = part.float()
    q = torch.randn(B, H * (D + P) + 8, generator=g).bfloat16()
    wuk, wuv = torch.randn(H * D, R, generator=g).bfloat16(), torch.randn(H * V, R, generator=g).bfloat16()
    sink, gate = torch.randn(H, generator=g), torch.randn(B, H * V, generator=g).bfloat16()
    qd, scale = q.cuda()[:, :H * (D + P)], (D + P) ** -0.5 * R ** -0.5
    qa = torch.full((B, H, W), float("nan"), device="cuda")
    k.latent_absorb(qd, wuk.cuda(), qa, H, D, P, R, scale)
    qh = q[:, :H * (D + P)].double().view(B, H, D + P)
    want = torch.cat([torch.einsum("bhd,hdr->bhr", qh[..., :D], wuk.double().view(H, D, R)), qh[..., D:]], -1) * scale
    assert float((qa.cpu().double() - want).abs().max()) < 2e-6 * D ** 0.5 * float(want.abs().max())
    ctx = SimpleNamespace(tok_pos=torch.tensor(lens, dtype=torch.int32).cuda() - 1, tok_seq=torch.arange(B, dtype=torch.int32).cuda())
    part = torch.full((B, H, n_split, R + 2), float("nan"), device="cuda")
    k.latent_attn(qa, pages.bfloat16().cuda(), ctx, table.cuda(), part, H, R, P, n_split, window=window)
    for mode, gt in ((0, None), (1, gate[:, :H]), (2, gate)):
        out = torch.full((B, H * V), float("nan"), dtype=torch.bfloat16, device="cuda")
        olat = torch.empty((B, H, R), device="cuda")
        k.latent_expand(part, olat, wuv.cuda(), out, H, V, R, n_split, sink=sink.cuda() if mode else None, gate=gt.cuda() if mode else None)
        lat = torch.empty(B, H, R, dtype=torch.float64)
        for b, n in enumerate(lens):
            seen = rows[b][max(0, n - window) if window else 0:].double()
            s = qa[b].cpu().double() @ seen.T
            w = torch.cat([s, sink.double()[:, None]], 1).softmax(-1)[:, :-1] if mode else s.softmax(-1)
            lat[b] = w @ seen[:, :R]
        assert float((olat.cpu().double() - lat).abs().max()) < 2e-6 * W ** 0.5 * float(lat.abs().max())
        want = torch.einsum("bhr,hvr->bhv", olat.cpu().double(), wuv.double().view(H, V, R))
        if mode:
            want = want * torch.sigmoid(gt.double()).view(B, H, -1)
        assert float((out.cpu().double() - want.reshape(B, -1)).abs().max()) < 2.0 ** -8 * float(want.abs().max())


@pytest.mark.parametrize("sink", [False, True])
def test_cached_latents_that_are_no_numbers_are_not_passed_over(sink):
    """A page of a row's keys is NaN and falls to a split of its own: the row's output is NaN, as with one split, and the other row's is not."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k, H, R, P, V = KernelSet(torch.bfloat16).mix, 3, 64, 16, 24
    g = torch.Generator().manual_seed(1)
    pages, table = torch.randn(10, 1, 64, R + P, generator=g).bfloat16(), torch.arange(10, dtype=torch.int32).view(2, 5)
    pages[2] = float("nan")
    qa, wuv = torch.randn(2, H, R + P, generator=g).cuda(), torch.randn(H * V, R, generator=g).bfloat16().cuda()
    ctx = SimpleNamespace(tok_pos=torch.tensor([300, 250], dtype=torch.int32).cuda(), tok_seq=torch.arange(2, dtype=torch.int32).cuda())
    for n_split in (1, 5):
        part = torch.zeros((2, H, n_split, R + 2), device="cuda")
        k.latent_attn(qa, pages.cuda(), ctx, table.cuda(), part, H, R, P, n_split)
        olat, out = torch.empty((2, H, R), device="cuda"), torch.empty((2, H * V), dtype=torch.bfloat16, device="cuda")
        k.latent_expand(part, olat, wuv, out, H, V, R, n_split, sink=torch.zeros(H, device="cuda") if sink else None)
        assert bool(out[0].isnan().all()) and bool(out[1].isfinite().all()), n_split


def test_sums_over_cached_latents_are_rounded_as_floats():
    """Many keys in one split: a sum that stayed on the tensor cores all the way, which cut where FMA rounds, would be 1.2e-5 off here.
    A page's sum is cut up to 12 times and a score 9 times in three groups, each by up to 2^-24 of its size at that step: (12 + 3) / 2 of
    them, 4.5e-7, and the roundings of the softmax."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k, B, H, R, P, n = KernelSet(torch.bfloat16).mix, 2, 16, 512, 64, 4096
    g = torch.Generator().manual_seed(2)
    pages, qa = torch.randn(B * n // 64, 1, 64, R + P, generator=g).bfloat16(), torch.randn(B, H, R + P, generator=g) / (R + P) ** 0.5
    table = torch.arange(B * n // 64, dtype=torch.int32).view(B, -1)
    ctx = SimpleNamespace(tok_pos=torch.full((B,), n - 1, dtype=torch.int32).cuda(), tok_seq=torch.arange(B, dtype=torch.int32).cuda())
    part, olat = torch.empty((B, H, 1, R + 2), device="cuda"), torch.empty((B, H, R), device="cuda")
    k.latent_attn(qa.cuda(), pages.cuda(), ctx, table.cuda(), part, H, R, P, 1)
    k.latent_expand(part, olat, torch.zeros(H * 8, R).bfloat16().cuda(), torch.empty((B, H * 8), dtype=torch.bfloat16, device="cuda"), H, 8, R, 1)
    keys = pages.view(B, n, R + P).double()
    want = torch.einsum("bhw,bnw->bhn", qa.double(), keys).softmax(-1) @ keys[..., :R]
    assert float((olat.cpu().double() - want).norm() / want.norm()) < 6e-7


def test_latent_weights_and_pages_at_any_place():
    """The decode form's matrices and pages two bytes off a multiple of 16: taken as before, by the kernels that ask for no alignment."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k, H, D, P, V, R, n = KernelSet(torch.bfloat16).mix, 4, 16, 8, 24, 64, 130
    g = torch.Generator().manual_seed(3)

    def off(*shape):
        t = torch.randn(math.prod(shape) + 1, generator=g).bfloat16().cuda()
        return t[1:].view(shape), t[1:].view(shape).clone()
    got = []
    for wuk, wuv, pages in zip(off(H * D, R), off(H * V, R), off(3, 1, 64, R + P)):
        q = torch.randn(1, H * (D + P), generator=torch.Generator().manual_seed(4)).bfloat16().cuda()
        ctx = SimpleNamespace(tok_pos=torch.tensor([n - 1], dtype=torch.int32).cuda(), tok_seq=torch.zeros(1, dtype=torch.int32).cuda())
        qa, part = torch.empty((1, H, R + P), device="cuda"), torch.empty((1, H, 2, R + 2), device="cuda")
        k.latent_absorb(q, wuk, qa, H, D, P, R, 0.2)
        k.latent_attn(qa, pages, ctx, torch.arange(3, dtype=torch.int32).view(1, 3).cuda(), part, H, R, P, 2)
        olat, out = torch.empty((1, H, R), device="cuda"), torch.empty((1, H * V), dtype=torch.bfloat16, device="cuda")
        k.latent_expand(part, olat, wuv, out, H, V, R, 2)
        got.append(out.float())
    assert float((got[0] - got[1]).abs().max()) <= 2.0 ** -7 * float(got[1].abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W, ld, off", [(8, 8, 0), (248, 504, 256), (2048, 4096, 2048), (4096, 4096, 0), (4104, 4104, 0), (2044, 2048, 0),
                                        (256, 516, 4), (1024, 1030, 0)])
@pytest.mark.parametrize("act", ["sigmoid", "silu"])
def test_gated_row_rms_at_its_widths(dtype, W, ld, off, act):
    """Eight elements a thread, and the widths and places that are not for it, against 64 bits: the output's rounding (2^-8 in
    bfloat16) and float sums and functions (2e-6)."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    g = torch.Generator().manual_seed(W)
    o, wide, w = torch.randn(5, W, generator=g), torch.randn(5, ld, generator=g).to(dtype), torch.rand(W, generator=g)
    gate, y = wide.cuda()[:, off:off + W], torch.full((5, W), float("nan"), dtype=dtype, device="cuda")
    KernelSet(dtype).mix.gated_row_rms(o.cuda(), gate, w.cuda(), y, 1e-6, act)
    z = wide[:, off:off + W].double()
    want = o.double() * torch.rsqrt((o.double() ** 2).mean(1, keepdim=True) + 1e-6) * w.double() * torch.sigmoid(z) * (z if act == "silu" else 1)
    assert bool(((y.cpu().double() - want).abs() <= (2 ** -8 if dtype == torch.bfloat16 else 2e-6) * want.abs() + 2e-6).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H, D, V, B", [(16, 128, 128, 9), (3, 10, 16, 1), (2, 250, 64, 300), (5, 64, 32, 40)])
def test_a_decode_step_of_linear_attention_walks_its_states(dtype, H, D, V, B):
    """One row a sequence, fewer pairs than blocks and several a block, slots out of order: states to one rounding of their two terms
    (1e-6 of the largest), outputs to float sums of D terms (1e-6 sqrt(D))."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k = KernelSet(dtype).mix
    g = torch.Generator().manual_seed(D)
    proj, state0 = torch.randn(B, 2 * H * D + H * V, generator=g).to(dtype), torch.randn(B + 2, H, D, V, generator=g)
    decay, slots = torch.rand(H, generator=g), torch.randperm(B + 2, generator=g)[:B].to(torch.int32)
    ctx = SimpleNamespace(seq_start=torch.arange(B + 1, dtype=torch.int32).cuda(), slots=slots.cuda(), n_seqs=B, max_new=1,
                          engine=SimpleNamespace(sm_count=148), err_flag=torch.zeros(1, dtype=torch.int32, device="cuda"))
    st, o = state0.clone().cuda(), torch.full((B, H * V), float("nan"), device="cuda")
    k.lin_attn_decay(proj.cuda(), 0, H * D, 2 * H * D, decay.cuda(), st, ctx, o, H, D, V)
    q, kk, v = (plain.silu(t).view(B, H, -1) for t in proj.double().split([H * D, H * D, H * V], 1))
    want, at = state0.double(), slots.long()
    want[at] = decay.double()[:, None, None] * want[at] + kk[..., None] * v[:, :, None]
    y = torch.einsum("bhdv,bhd->bhv", want[at], q).reshape(B, -1)
    assert int(ctx.err_flag) == 0
    assert float((st.cpu().double() - want).abs().max()) < 1e-6 * float(want.abs().max())
    assert float((o.cpu().double() - y).abs().max()) < 1e-6 * D ** 0.5 * float(y.abs().max())


STEP_GIVES_UP = """
#include "state_step.cuh"
struct Job {
  float *state, *y; int H, N, V;
  __device__ int heads() const { return H; }
  __device__ int rows() const { return N; }
  __device__ int cols() const { return V; }
  __device__ float* place(int b, int h) const { return state + (size_t)(b * H + h) * N * V; }
  __device__ void fetch(step::Row& r, int, int, int) const { r.b = r.c = r.x = r.d = 1.f; r.dec = 0.5f; }
  __device__ void finish(int b, int h, int v, float s, float, float) const { y[(b * H + h) * V + v] = s; }
};
extern "C" int run(float* state, float* y, int B, int H, int N, int V, int* err, cudaStream_t stream) {
  return step::launch(Job{state, y, H, N, V}, N, V, B * H, 1, err, stream);      // "one SM": two blocks that stay
}
"""


def test_a_state_whose_wait_runs_out_is_left_as_it_was(tmp_path):
    """The walk over the states, built with one thread's wait for a block's third pair counted as run out: the two pairs in front of it
    are advanced and stored, none behind it is, the error flag is raised and the stream goes on."""
    import ctypes
    import subprocess
    from scriptling_llm_lib_b200.csrc import build
    for f in ("common.cuh", "tcgen05.cuh"):
        (tmp_path / f).write_text((build.CSRC / f).read_text())
    wait = "if (!mbar_wait(full + 8 * (i % RING), (i / RING) & 1, abort)) ok = false;"
    walk = (build.CSRC / "state_step.cuh").read_text()
    assert walk.count(wait) == 1
    (tmp_path / "state_step.cuh").write_text(walk.replace(wait, wait + " if (i == 2 && threadIdx.x == 7) ok = false;"))
    (tmp_path / "t.cu").write_text(STEP_GIVES_UP)
    subprocess.run([build.find_nvcc(), *build.ARCH_FLAGS, *build.NVCC_FLAGS, "-I", str(tmp_path), "-o", str(tmp_path / "t.so"), str(tmp_path / "t.cu")],
                   check=True, capture_output=True, timeout=300)
    lib = ctypes.CDLL(str(tmp_path / "t.so"))
    B, H, N, V = 3, 5, 40, 64
    state0 = torch.randn(B, H, N, V, generator=torch.Generator().manual_seed(1))
    st, y, err = state0.cuda(), torch.zeros(B, H, V, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())      # noqa: E731
    assert lib.run(p(st), p(y), B, H, N, V, p(err), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    want = state0.view(B * H, N, V).clone()
    want[:4] = 0.5 * want[:4] + 1                    # two blocks: pairs 0, 2, ... and 1, 3, ...; the third of either gives up
    assert int(err) == 5
    assert torch.equal(st.view(B * H, N, V)[4:].cpu(), want[4:])
    assert float((st.view(B * H, N, V)[:4].cpu() - want[:4]).abs().max()) < 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("inner, N, lens", [(100, 16, [1, 63, 64, 65, 200]), (256, 5, [300]), (130, 17, [16, 33, 112]), (64, 32, [129, 2]),
                                            (4096, 1, [2100])])
def test_selective_scan_in_pieces_against_the_recurrence(dtype, inner, N, lens):
    """Runs around the pieces' lengths (16, 32 and 64 rows by the size of the step), channels that fill no block, every built number of
    states and ones between; states that are not zero, slots out of order; some decays near 1, some total. The states, float sums
    decayed along the run, to 2e-6 sqrt(rows) of the largest; outputs to that and their own rounding."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k = KernelSet(dtype).mix
    g = torch.Generator().manual_seed(inner + N)
    T, K, slots = sum(lens), 3, list(range(len(lens)))[::-1]
    xz = torch.randn(T, 2 * inner, generator=g).to(dtype)
    bc = torch.randn(T, K + 2 * N, generator=g).to(dtype)
    raw = torch.randn(T, inner, generator=g) * 2 - 3
    bias, d = torch.randn(inner, generator=g), torch.randn(inner, generator=g)
    a_log = torch.randn(inner, N, generator=g) * 2
    start = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    state0 = torch.randn(len(lens) + 1, inner, N, generator=g)
    ctx = SimpleNamespace(seq_start=torch.from_numpy(start).cuda(), slots=torch.tensor(slots, dtype=torch.int32).cuda(),
                          n_seqs=len(lens), max_new=max(lens), engine=SimpleNamespace(sm_count=148))
    k.scan_pays = lambda *a: True
    st, xd = state0.clone().cuda(), xz.cuda()
    out = torch.full((T, inner), float("nan"), dtype=dtype, device="cuda")
    k.selective_scan(xd[:, :inner], raw.cuda(), bias.cuda(), a_log.cuda(), d.cuda(), bc.cuda(), K, K + N, xd[:, inner:], st, ctx, out, inner, N)
    x, z, (_, B, C) = xz[:, :inner].double(), xz[:, inner:].double(), bc.double().split([K, N, N], 1)
    dt = torch.nn.functional.softplus(raw.double() + bias.double(), threshold=1e9)
    A, want, after = -torch.exp(a_log.double()), torch.empty(T, inner, dtype=torch.float64), state0.double()
    for b, slot in enumerate(slots):
        S = state0[slot].double()
        for t in range(start[b], start[b + 1]):
            S = torch.exp(dt[t, :, None] * A) * S + (dt[t] * x[t])[:, None] * B[t]
            want[t] = (S @ C[t] + d.double() * x[t]) * plain.silu(z[t])
        after[slot] = S
    assert float((st.cpu().double() - after).abs().max()) < 2e-6 * max(lens) ** 0.5 * float(after.abs().max())
    tol = 2e-6 * max(lens) ** 0.5 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    assert float((out.cpu().double() - want).abs().max()) < tol * float(want.abs().max())
    assert torch.equal(st[len(lens)].cpu(), state0[len(lens)])          # a slot no sequence of the step holds is left alone


@pytest.mark.parametrize("H, D, V, pad", [(2, 128, 128, 0), (3, 24, 40, 0), (1, 64, 200, 8), (2, 50, 70, 3)])
def test_linear_attention_in_chunks_against_the_recurrence(H, D, V, pad):
    """Runs of one row to three chunks in one step, from states that are not zero, slots out of order; widths that fill the tiles, that
    leave them partly empty, and that allow no 16-byte access; decays of 0, 1 and between. Float sums of up to 300 terms in three
    bfloat16 parts: 1e-5 of the largest element."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k = KernelSet(torch.bfloat16).mix
    g = torch.Generator().manual_seed(D)
    lens = [1, 127, 128, 129, 300, 16]
    T, slots = sum(lens), [5, 0, 3, 1, 6, 2]
    proj = torch.randn(T, 2 * H * D + H * V + pad, generator=g).bfloat16()
    decay = torch.tensor([[0.97], [0.0, 1.0], [0.3, 0.995, 1.0]][H - 1])
    start = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    state0 = torch.randn(len(lens) + 2, H, D, V, generator=g)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(seq_start=torch.from_numpy(start).cuda(), slots=torch.tensor(slots, dtype=torch.int32).cuda(), err_flag=err,
                          n_seqs=len(lens), max_new=max(lens), engine=SimpleNamespace(sm_count=148))
    st = state0.clone().cuda()
    o = torch.full((T, H * V), float("nan"), dtype=torch.float32, device="cuda")
    k.chunk.lin_attn(proj.cuda(), 0, H * D, 2 * H * D, decay.cuda(), st, ctx, o, H, D, V)
    q, kk, v = (plain.silu(t).view(T, H, -1) for t in proj[:, :2 * H * D + H * V].double().split([H * D, H * D, H * V], 1))
    want, after = torch.empty((T, H, V), dtype=torch.float64), state0.double()
    for b, slot in enumerate(slots):
        S = state0[slot].double()
        for t in range(start[b], start[b + 1]):
            S = decay.double()[:, None, None] * S + kk[t, :, :, None] * v[t, :, None]
            want[t] = torch.einsum("hdv,hd->hv", S, q[t])
        after[slot] = S
    assert int(err) == 0
    assert float((o.cpu().double() - want.view(T, -1)).abs().max()) < 1e-5 * float(want.abs().max())
    assert float((st.cpu().double() - after).abs().max()) < 1e-5 * float(after.abs().max())
    assert torch.equal(st[4].cpu(), state0[4])          # a slot no sequence of the step holds is left alone


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["query", "key", "value", "state"])
def test_what_is_not_finite_in_a_row_stays_behind_it_in_chunks(where, bad):
    """One element that is not finite, in rows of the first, a middle and the last chunk: what is not finite behind it is what the
    recurrence in 64 bits leaves so, element by element, and the rest agrees with it."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k, H, D, V, lens, slots = KernelSet(torch.bfloat16).mix, 2, 24, 40, [300, 140, 257], [2, 0, 3]
    start, decay = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32), torch.tensor([0.9, 0.99])
    for at in (5, 131, 299, 300 + 127, 440 + 200):
        g = torch.Generator().manual_seed(at)
        proj, state0 = torch.randn(sum(lens), 2 * H * D + H * V, generator=g).bfloat16(), torch.randn(4, H, D, V, generator=g)
        if where == "state":
            state0[2, 1, 3, 5] = bad
        else:
            proj[at, {"query": D + 7, "key": H * D + D + 7, "value": 2 * H * D + V + 3}[where]] = bad
        ctx = SimpleNamespace(seq_start=torch.from_numpy(start).cuda(), slots=torch.tensor(slots, dtype=torch.int32).cuda(), n_seqs=len(lens),
                              max_new=max(lens), err_flag=torch.zeros(1, dtype=torch.int32, device="cuda"))
        st, o = state0.clone().cuda(), torch.zeros(sum(lens), H * V, device="cuda")
        k.chunk.lin_attn(proj.cuda(), 0, H * D, 2 * H * D, decay.cuda(), st, ctx, o, H, D, V)
        q, kk, v = (plain.silu(t).view(sum(lens), H, -1) for t in proj.double().split([H * D, H * D, H * V], 1))
        want, after = torch.empty((sum(lens), H, V), dtype=torch.float64), state0.double()
        for b, slot in enumerate(slots):
            S = state0[slot].double()
            for t in range(start[b], start[b + 1]):
                S = decay.double()[:, None, None] * S + kk[t, :, :, None] * v[t, :, None]
                want[t] = torch.einsum("hdv,hd->hv", S, q[t])
            after[slot] = S
        assert int(ctx.err_flag) == 0 and not bool(want.isfinite().all())
        for a, b in ((want.view(sum(lens), -1), o.cpu()), (after, st.cpu())):
            both = a.isfinite()
            assert torch.equal(both, b.isfinite()), (where, at, (both != b.isfinite()).nonzero()[:4])
            assert float((a[both] - b[both]).abs().max()) < 1e-5 * float(a[both].abs().max())


def test_linear_attention_in_chunks_over_long_runs():
    """Runs of up to eleven chunks, past the eight that the hand-over asks for at a time, beside one of a row: 1e-5 of the largest element
    as for short runs."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k, H, D, V, lens, slots = KernelSet(torch.bfloat16).mix, 2, 24, 40, [1, 1025, 1300, 640], [3, 0, 4, 1]
    g, T = torch.Generator().manual_seed(8), sum(lens)
    proj, decay, state0 = torch.randn(T, 2 * H * D + H * V, generator=g).bfloat16(), torch.tensor([0.9995, 0.97]), torch.randn(5, H, D, V, generator=g)
    start = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ctx = SimpleNamespace(seq_start=torch.from_numpy(start).cuda(), slots=torch.tensor(slots, dtype=torch.int32).cuda(), n_seqs=4, max_new=1300)
    st, o = state0.clone().cuda(), torch.full((T, H * V), float("nan"), device="cuda")
    k.chunk.lin_attn(proj.cuda(), 0, H * D, 2 * H * D, decay.cuda(), st, ctx, o, H, D, V)
    q, kk, v = (plain.silu(t).view(T, H, -1) for t in proj.double().split([H * D, H * D, H * V], 1))
    want, after = torch.empty((T, H, V), dtype=torch.float64), state0.double()
    for b, slot in enumerate(slots):
        S = state0[slot].double()
        for t in range(start[b], start[b + 1]):
            S = decay.double()[:, None, None] * S + kk[t, :, :, None] * v[t, :, None]
            want[t] = torch.einsum("hdv,hd->hv", S, q[t])
        after[slot] = S
    assert float((o.cpu().double() - want.view(T, -1)).abs().max()) < 1e-5 * float(want.abs().max())
    assert float((st.cpu().double() - after).abs().max()) < 1e-5 * float(after.abs().max())


def test_silu_of_every_bfloat16_in_the_chunks():
    """One row, values of every finite bfloat16 there is: the state silu(k) silu(v) to a float's few last places (its parts, down to where
    they leave float's range: 1e-4 below 1e-30), and what silu makes 0 is 0."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    k, D = KernelSet(torch.bfloat16).mix, 8
    v = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    v = v[v.isfinite() & (v.abs() < 1e30)]
    v = v[:len(v) // 8 * 8]
    V, key = len(v), torch.tensor(1.28).bfloat16()
    proj = torch.cat([torch.ones(D).bfloat16(), key.expand(D), v])[None].cuda()
    ctx = SimpleNamespace(seq_start=torch.tensor([0, 1], dtype=torch.int32).cuda(), slots=torch.zeros(1, dtype=torch.int32).cuda(), n_seqs=1, max_new=1)
    st, o = torch.zeros(1, 1, D, V, device="cuda"), torch.empty(1, V, device="cuda")
    k.chunk.lin_attn(proj, 0, D, 2 * D, torch.ones(1, device="cuda"), st, ctx, o, 1, D, V)
    want = plain.silu(key.double()) * torch.where(v.double() < -700, torch.zeros(V, dtype=torch.float64), plain.silu(v.double().clamp(min=-700)))
    err = (st[0, 0, 0].cpu().double() - want).abs()
    tol = torch.where(want.abs() > 1e-30, 1e-6, 1e-4) * want.abs() + 1e-36
    assert bool((err <= tol).all()), (v[err > tol][:8], err[err > tol][:8])


def test_heads_of_linear_attention_in_several_passes(monkeypatch):
    """As many heads at a time as the scratch's bound holds: three, then two; the bits of all five at once."""
    from scriptling_llm_lib_b200.csrc.bindings import ChunkKernels, KernelSet
    k, H, D, V, lens = KernelSet(torch.bfloat16).mix, 5, 24, 136, [300, 140]
    g = torch.Generator().manual_seed(6)
    proj, decay = torch.randn(sum(lens), 2 * H * D + H * V, generator=g).bfloat16().cuda(), torch.rand(H, generator=g).cuda()
    state0, got = torch.randn(2, H, D, V, generator=g), []
    ctx = SimpleNamespace(seq_start=torch.tensor([0, 300, 440], dtype=torch.int32).cuda(), slots=torch.tensor([1, 0], dtype=torch.int32).cuda(), n_seqs=2,
                          max_new=300)
    for bound in (ChunkKernels.SCRATCH_BYTES, (sum(lens) // 128 + 2) * 3 * 4 * D * V):
        monkeypatch.setattr(ChunkKernels, "SCRATCH_BYTES", bound)
        st, o = state0.clone().cuda(), torch.full((sum(lens), H * V), float("nan"), device="cuda")
        k.chunk.lin_attn(proj, 0, H * D, 2 * H * D, decay, st, ctx, o, H, D, V)
        got.append((st, o))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_the_norm_adds_a_normed_addend_and_keeps_the_sum():
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    for dtype in (torch.float32, torch.bfloat16):
        k = KernelSet(dtype).mix
        g = torch.Generator().manual_seed(5)
        x = torch.randn(9, 50, generator=g)
        parts = torch.randn(3, 9, 50, generator=g)
        pw, pb, w, b = (torch.randn(50, generator=g) for _ in range(4))
        want_x = x.double() + torch.tanh(0.7 * parts.double().sum(0)) * pw.double() + pb.double()
        want = torch.tanh(1.3 * want_x) * w.double() + b.double()
        xd = x.clone().cuda()
        out = torch.empty((9, 50), dtype=dtype, device="cuda")
        k.dyt_add_norm(xd, parts.cuda(), (pw.cuda(), pb.cuda(), 0.7), None, w.cuda(), b.cuda(), 1.3, out)
        assert float((xd.cpu().double() - want_x).abs().max()) < 1e-5
        assert float((out.cpu().double() - want).abs().max()) < (1e-5 if dtype == torch.float32 else 3e-2)
        rows = torch.tensor([7, 2], dtype=torch.int32).cuda()
        x2 = x.clone().cuda()
        out2 = torch.empty((2, 50), dtype=dtype, device="cuda")
        one = parts[0].to(dtype)
        k.dyt_add_norm(x2, one.cuda(), None, rows, w.cuda(), b.cuda(), 1.3, out2)
        want2 = torch.tanh(1.3 * (x.double() + one.double())[[7, 2]]) * w.double() + b.double()
        assert torch.equal(x2.cpu(), x)                  # picked rows: the stream is left as it was
        assert float((out2.cpu().double() - want2).abs().max()) < (1e-5 if dtype == torch.float32 else 3e-2)


@pytest.mark.parametrize("T, top, E, pad", [(1, 1, 1, 1), (5, 3, 7, 256), (2048, 6, 64, 256), (700, 4, 1500, 1), (333, 8, 1025, 128), (900, 2, 8192, 1)])
def test_moe_grouping_gives_every_pair_its_row(T, top, E, pad):
    """Offsets, tiles and rows of the grouped pairs, a share of the pairs a block of the cluster: few pairs, more experts than threads,
    experts without a pair; then the rows that gathering by them leaves, and their products on either tile."""
    k = KernelSet(torch.bfloat16)
    g = torch.Generator().manual_seed(T)
    idx = torch.stack([torch.randperm(E, generator=g)[:top] if E < 2000 else torch.randint(0, E, (top,), generator=g) for _ in range(T)]).int()
    idx[:, 0] = torch.where(torch.rand(T, generator=g) < 0.3, idx[0, 0], idx[:, 0])
    pairs, counts = T * top, torch.bincount(idx.flatten().long(), minlength=E)
    rows = pairs if pad == 1 else -(-(pairs + E * (pad - 1)) // pad) * pad
    offsets, rop = torch.full((E + 1,), -7, dtype=torch.int32, device="cuda"), torch.full((pairs,), -7, dtype=torch.int32, device="cuda")
    por, tiles = torch.full((rows,), -7, dtype=torch.int32, device="cuda"), torch.full((max(1, rows // pad),), -7, dtype=torch.int32, device="cuda")
    k.mix.moe_group_rows(idx.cuda(), E, offsets, por, rop, tiles if pad > 1 else None, pad=pad)
    want = torch.cat([torch.zeros(1, dtype=torch.long), ((counts + pad - 1) // pad * pad).cumsum(0)])
    assert torch.equal(offsets.cpu().long(), want)
    row, experts = rop.cpu().long(), idx.flatten().long()
    assert torch.equal(por.cpu().long()[row], torch.arange(pairs)) and row.unique().numel() == pairs
    assert bool(((row >= want[experts]) & (row < want[experts] + counts[experts])).all())
    if pad > 1:
        first = torch.arange(rows // pad) * pad
        assert torch.equal(tiles.cpu().long(), (torch.searchsorted(want[1:], first, right=True)).clamp(max=E - 1))
    if pad == 1 or E > 100:
        return
    K, N, tc, flag = 72, 264, k.tensor_core, torch.zeros(1, dtype=torch.int32, device="cuda")
    h, w = torch.randn(T, K, generator=g).bfloat16().cuda(), (torch.randn(E, N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    xs = torch.full((rows, K), float("nan"), dtype=torch.bfloat16, device="cuda")
    k.mix.moe_spread_rows(h, rop, top, xs)
    assert torch.equal(xs[rop.long()], h.repeat_interleave(top, 0))
    out = torch.full((rows, N), 7.0, device="cuda")
    tc.gemm_grouped(xs, w, out, tiles, flag, rows_used=offsets[E:], tile_rows=pad)
    exact = torch.einsum("pk,pnk->pn", xs[rop.long()].double(), w.double()[experts.cuda()])
    got = out[rop.long()].double()
    assert ((got - exact).norm() / exact.norm()).item() < 2e-6 and int(flag) == 0       # products of bfloat16, float sums of 72 terms
    assert bool((out[int(want[-1]):] == 7.0).all())                                     # tiles behind the rows in use are left alone


def test_experts_one_by_one_and_grouped_agree(folders):
    """A step of few rows runs every (token, expert) pair by itself, a longer one groups them by expert."""
    folder, cfg, W = folders["A"]
    tokens = ids(80, cfg["vocab"], 18)
    eng = engine(folder)
    whole = run(eng, [tokens])                       # 80 rows x 2 experts: grouped
    small = run(eng, cut(tokens, [7] * 12))          # 7 rows a step: one by one
    assert rel(small, whole) < TOL_F32


# --------------------------------------------------------------------------- the entry point
def test_greedy_generation_through_the_entry_point(folders):
    from scriptling_llm_lib_b200 import llm
    folder, cfg, W = folders["A"]
    prompt = ids(21, cfg["vocab"], 19)
    for dtype in ("float32", "bfloat16"):
        out = llm.generate(str(folder), prompt, max_tokens=12, strategy="greedy", dtype=dtype)
        tokens = list(prompt)
        for t in out:
            lg = plain_logits(cfg, W, tokens)[-1]
            top2 = lg.topk(2).values
            if dtype == "float32" or float(top2[0] - top2[1]) > 0.2 * float(lg.abs().max()):
                assert int(lg.argmax()) == t
            tokens.append(t)
        assert len(out) == 12


def test_random_weights_mode_and_the_command_line(tmp_path):
    import subprocess
    import sys
    from pathlib import Path
    cfg_path = tmp_path / "config.json"
    cfg_path.write_text(json.dumps(CFG_B))
    eng = engine(f"random:{cfg_path}:3", "bfloat16")
    got = run(eng, [ids(40, CFG_B["vocab"], 1)])
    assert torch.isfinite(got).all() and float(got.abs().max()) > 0
    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-m", "scriptling_llm_lib_b200", "-model", f"random:{cfg_path}:3", "-prompt", "1,2,3",
                        "-tokens", "4"], cwd=root, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
