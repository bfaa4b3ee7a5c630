"""Which kernel a step runs on, by its sizes (no GPU: the launches are recorded, not made)."""
from types import SimpleNamespace

import pytest
import torch

from scriptling_llm_lib_b200.csrc.bindings import ChunkKernels, MixKernels, SequenceKernels


def _recorded(cls, walk):
    """A set of kernels whose chunked and walked forms only say which of them ran."""
    k, ran = cls.__new__(cls), []
    k.dtype, k._fns = torch.bfloat16, {}
    k._chunk = SimpleNamespace(delta=lambda *a: ran.append("chunks"), lin_attn=lambda *a: ran.append("chunks"))
    setattr(k, walk, lambda *a: ran.append("walk"))
    return k, ran


def _ctx(lens):
    return SimpleNamespace(n_seqs=len(lens), max_new=max(lens), engine=SimpleNamespace(sm_count=148))


# measured: walked / in chunks, us
DELTA = [(16, 128, [2048], "chunks"),                    # 639 / 173
         (16, 128, [200] * 8, "chunks"),                 # 261 / 167
         (16, 128, [128], "walk"),                       # 49 / 63
         (16, 128, [192] + [16] * 100, "walk"),          # 504 / 1,036
         (16, 128, [1000] + [32] * 64, "walk"),          # 639 / 774
         (2, 128, [1000] + [32] * 64, "chunks"),         # 308 / 116
         (4, 128, [192] + [4] * 16, "walk"),             # 66 / 71
         (16, 64, [192] + [32] * 200, "walk"),           # 536 / 1,407
         (16, 16, [200] * 8, "walk"),                    # 67 / 108
         (64, 16, [192] + [16] * 100, "walk"),           # 170 / 2,343
         (64, 16, [2048], "chunks")]                     # 595 / 398


@pytest.mark.parametrize("H, d, lens, want", DELTA)
def test_the_delta_rule_goes_in_chunks_where_that_is_faster(H, d, lens, want):
    k, ran = _recorded(SequenceKernels, "delta_walk")
    T = sum(lens)
    f = lambda *s: torch.empty(s, device="meta")      # noqa: E731
    k.delta_rule(f(T, 2 * H * d), f(T, H * d), f(T, 3 * H), f(len(lens), H, d, d), _ctx(lens), f(T, H * d), H, H, d, d)
    assert ran == [want]


LINEAR = [(16, 128, [2048], "chunks"),                   # 459 / 78
          (16, 128, [144], "chunks"),                    # 47 / 39
          (16, 128, [144] + [16] * 100, "walk"),         # 488 / 735
          (16, 128, [1000] + [32] * 64, "walk"),         # 444 / 542
          (2, 128, [144] + [16] * 100, "walk"),          # 66 / 80
          (16, 64, [144] + [4] * 16, "walk"),            # 50 / 63
          (16, 16, [192], "walk"),                       # 27 / 29
          (16, 16, [512], "chunks"),                     # 65 / 29
          (16, 16, [200] * 8, "walk"),                   # 34 / 53
          (64, 16, [1000] + [32] * 64, "walk")]          # 161 / 950


@pytest.mark.parametrize("H, d, lens, want", LINEAR)
def test_linear_attention_goes_in_chunks_where_that_is_faster(H, d, lens, want):
    k, ran = _recorded(MixKernels, "lin_attn_walk")
    T = sum(lens)
    f = lambda *s: torch.empty(s, device="meta")      # noqa: E731
    k.lin_attn_decay(f(T, 3 * H * d), 0, H * d, 2 * H * d, f(H), f(len(lens), H, d, d), _ctx(lens), f(T, H * d), H, d, d)
    assert ran == [want]


SCAN = [(4096, 16, [2048], "pieces"),                    # 466 / 143
        (4096, 16, [64], "walk"),                        # 18 / 21
        (256, 16, [300], "pieces"),                      # 56 / 21
        (4096, 16, [96] + [4] * 16, "pieces"),           # 67 / 45
        (1024, 16, [96] + [4] * 16, "walk"),             # 24 / 26
        (1024, 32, [96] + [4] * 16, "walk"),             # 29 / 41
        (64, 16, [96] + [16] * 100, "walk"),             # 21 / 24
        (512, 4, [96] + [16] * 100, "walk"),             # 22 / 26
        (1024, 16, [96] + [16] * 100, "pieces"),         # 132 / 70
        (4096, 33, [2048], "walk"),                      # more states than it is built for
        (4096, 16, [96] + [16] * 2000, "walk")]          # a state for each of so many runs would take 550 MB


@pytest.mark.parametrize("inner, N, lens, want", SCAN)
def test_the_selective_scan_goes_in_pieces_where_that_is_faster(monkeypatch, inner, N, lens, want):
    from scriptling_llm_lib_b200.csrc import bindings
    k, ran = MixKernels.__new__(MixKernels), []
    k.dtype = torch.bfloat16
    k._fn = lambda name: lambda *a: ran.append(name) or 0
    monkeypatch.setattr(bindings, "_ptr", lambda *a: None)
    monkeypatch.setattr(bindings, "_stream", lambda: None)
    k._view = lambda *a: None
    T, ctx = sum(lens), _ctx(lens)
    ctx.seq_start = ctx.slots = None
    f = lambda *s, dt=torch.bfloat16: torch.empty(s, device="meta", dtype=dt)      # noqa: E731
    f32 = torch.float32
    k.selective_scan(f(T, inner), f(T, inner, dt=f32), f(inner), f(inner, N), f(inner), f(T, 2 * N), 0, N, f(T, inner),
                     f(len(lens), inner, N, dt=f32), ctx, f(T, inner), inner, N)
    assert ran == ["selective_scan_pieces" if want == "pieces" else "selective_scan"]


@pytest.mark.parametrize("D, V, rows, from_start, want", [(64, 128, 8, True, False), (64, 128, 16, True, False), (64, 128, 17, True, True),
                                                          (64, 128, 1, False, True), (32, 32, 2, True, False), (32, 32, 4, True, True),
                                                          (80, 80, 1, True, False), (80, 80, 2, True, True), (80, 80, 2, False, True),
                                                          (72, 72, 16, True, False), (200, 128, 500, True, False)])
def test_a_prompt_of_very_few_rows_keeps_the_kernels_without_tiles(D, V, rows, from_start, want):
    from scriptling_llm_lib_b200.parts.attention import exact_prompt_kernel
    ctx = SimpleNamespace(is_decode=False, from_start=from_start, max_new=rows)
    assert exact_prompt_kernel(ctx, torch.bfloat16, D, V) == want
    assert not exact_prompt_kernel(ctx, torch.float32, D, V)
    ctx.is_decode = True
    assert not exact_prompt_kernel(ctx, torch.bfloat16, D, V)


def test_more_key_rows_than_a_tensor_map_reaches_keep_the_other_kernels():
    """A cache of narrow heads can hold more rows than the tcgen05 launcher takes: such a prompt is not refused but runs as before."""
    from scriptling_llm_lib_b200.parts.attention import Attention
    ran, H, D = [], 8, 16
    seen = lambda name: lambda *a, **k: ran.append(name)      # noqa: E731
    layer = Attention(128, H, H, D, None, "q", "k", "v", "o")
    ctx = SimpleNamespace(is_decode=False, from_start=True, max_new=100, n_seqs=1, seq_start=None, seq_pos0=None, err_flag=None,
                          kernels=SimpleNamespace(attn_paged=seen("paged"), prefill_attention_tc=SimpleNamespace(attn=seen("tcgen05"))))
    x = torch.empty((100, 128), dtype=torch.bfloat16, device="meta")
    for pages in (2 ** 31 // (H * 64) - 1, 2 ** 31 // (H * 64)):
        kp = torch.empty((pages, H, 64, D), dtype=torch.bfloat16, device="meta")
        layer._attend(torch.empty((100, 3 * H * D), dtype=torch.bfloat16, device="meta"), x, ctx, kp, kp, None, False, None, True)
    assert ran == ["tcgen05", "paged"]


@pytest.mark.parametrize("rows, n_seqs, H", [(2048, 1, 16), (16384, 1, 16), (16384, 8, 64), (12992, 401, 16), (16384, 1, 1), (130000, 1000, 32)])
def test_scratch_of_the_chunks_is_bounded(rows, n_seqs, H):
    """Heads are gone through as many at a time as the bound holds, evenly; one at least."""
    n, per = rows // ChunkKernels.CHUNK + n_seqs, ChunkKernels.DELTA_BYTES
    held = ChunkKernels.heads_held(n, H, per)
    passes = -(-H // held)
    assert 1 <= held <= H and (n * held * per <= ChunkKernels.SCRATCH_BYTES or held == 1)
    assert passes == 1 or n * -(-H // (passes - 1)) * per > ChunkKernels.SCRATCH_BYTES       # no pass more than it takes


def test_the_reserve_counts_what_a_recurrence_takes_beside_its_rows():
    """What the cache leaves free for a prompt step holds the chunks' scratch, alone and inside a parallel mixer."""
    from scriptling_llm_lib_b200.engine import Engine
    from scriptling_llm_lib_b200.parts.base import MIXERS, Norm, PartSpec
    delta = PartSpec("gated_delta_rule", dict(hidden=1024, n_heads=64, n_kv_heads=64, key_dim=16, value_dim=16, conv_taps=4, norm_eps=1e-6,
                                              **{n: n for n in ("q_name", "k_name", "v_name", "q_conv_name", "k_conv_name", "v_conv_name", "beta_name",
                                                                "decay_name", "a_log_name", "dt_bias_name", "gate_name", "norm_name", "o_name")}))
    eng = lambda parts: SimpleNamespace(layout=SimpleNamespace(hidden_size=1024, vocab_size=512), model=SimpleNamespace(parts=lambda: parts),      # noqa: E731
                                        PROMPT_TOKENS_PER_STEP=Engine.PROMPT_TOKENS_PER_STEP)
    plain = Engine.activation_reserve_bytes(eng([Norm(), object()]))
    for part in (MIXERS.build(delta), MIXERS.build(PartSpec("parallel", dict(branches=[("a", delta, 1.0)])))):
        assert Engine.activation_reserve_bytes(eng([Norm(), part])) == plain + ChunkKernels.SCRATCH_BYTES
    scan = PartSpec("selective_scan", dict(hidden=1024, inner=2048, n_state=16, dt_rank=64, conv_taps=4, **{n: n for n in (
        "in_name", "conv_name", "conv_bias_name", "x_name", "dt_name", "dt_bias_name", "a_log_name", "d_name", "o_name")}))
    rows = Engine.PROMPT_TOKENS_PER_STEP
    need = 4 * 2048 * (rows + (rows // 64 + 50) * 17)
    assert Engine.activation_reserve_bytes(eng([MIXERS.build(scan)])) >= plain + need
    assert MixKernels.scan_scratch_bytes(rows, 50, 2048, 16, 148) == need


@pytest.mark.parametrize("pairs, E, F, hidden, want", [(12288, 64, 1408, 2048, 256), (7168, 64, 1408, 2048, 128), (7169, 64, 1408, 2048, 256), (9000, 8, 64, 2048, 128),
                                                       (9000, 8, 65, 2048, 256), (9000, 8, 1408, 128, 128)])
def test_rows_of_a_tile_of_the_grouped_products(pairs, E, F, hidden, want):
    """256 rows on two SMs from more than 112 rows an expert on, where both products have more than 128 columns (gated: 2 F and hidden)."""
    from scriptling_llm_lib_b200.parts.experts import RoutedExperts
    part = RoutedExperts(hidden, F, E, 1, 1, 1, 1.0, "r", "c", [f"u{j}" for j in range(E)], [f"d{j}" for j in range(E)], act="silu_glu",
                         gate_names=[f"g{j}" for j in range(E)])
    assert part._tile_rows(pairs) == want


@pytest.mark.parametrize("D, V, decode, want", [(64, 128, True, "split"), (12, 20, True, "split"), (64, 126, True, "wide"), (64, 128, False, "wide"),
                                                (80, 80, True, "paged"), (24, 24, True, "split")])
def test_a_decode_step_of_unequal_widths_splits_its_keys(D, V, decode, want):
    """Widths in multiples of four: keys split over blocks; others, and the few rows of a portion, a block a row and head."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    from scriptling_llm_lib_b200.parts.attention import Attention
    ran, H, G = [], 8, 2
    seen = lambda name: lambda *a, **k: ran.append(name)      # noqa: E731
    layer = Attention(128, H, G, D, None, "q", "k", "v", "o", v_dim=V)
    kernels = SimpleNamespace(attn_paged=seen("paged"), attn_decode_split=seen("split"), seq=SimpleNamespace(attn_wide_value=seen("wide")),
                              attn_decode_split_takes=KernelSet.attn_decode_split_takes if D != 80 else lambda *a: False,
                              attn_decode_splits=KernelSet.attn_decode_splits)
    ctx = SimpleNamespace(is_decode=decode, from_start=False, max_new=1 if decode else 3, n_seqs=3, seq_pos0=None, seq_start=None, tok_pos=None,
                          tok_seq=None, kernels=kernels, pages_seen=lambda unit: 9, engine=SimpleNamespace(sm_count=148))
    x, kp = torch.empty((3, 128), dtype=torch.float32, device="meta"), torch.empty((9, G, 64, D), dtype=torch.float32, device="meta")
    layer._attend(torch.empty((3, H * D + G * (D + V)), dtype=torch.float32, device="meta"), x, ctx, kp, kp, None, False, None, True, 0)
    assert ran == [want]


@pytest.mark.parametrize("dtype, graphs, times", [(torch.bfloat16, True, 0), (torch.float32, False, 1), (torch.float32, True, 2)])
def test_the_reserve_counts_the_planes_where_a_matrix_is_kept_in_32_bit(dtype, graphs, times):
    """A bfloat16 engine's cache does not give way to products that it does not run; a captured decode step holds its own planes."""
    from scriptling_llm_lib_b200.csrc.bindings import SplitGemm
    from scriptling_llm_lib_b200.engine import Engine
    from scriptling_llm_lib_b200.parts.base import FeedForward, Norm
    from scriptling_llm_lib_b200.parts.linear import Linear

    def reserve(parts):
        return Engine.activation_reserve_bytes(SimpleNamespace(layout=SimpleNamespace(hidden_size=1024, vocab_size=512), use_graphs=graphs,
                                                               model=SimpleNamespace(parts=lambda: parts),
                                                               PROMPT_TOKENS_PER_STEP=Engine.PROMPT_TOKENS_PER_STEP))

    plain, outer, inner, lin = reserve([Norm(), object()]), FeedForward(), FeedForward(), Linear(["w"], [64], 128)
    outer.shared, inner.gates = inner, [Linear(["v"], [8], 8), lin]
    assert reserve([outer]) == plain == Engine.PROMPT_TOKENS_PER_STEP * 64 * 1024 + 4 * 512 * 4 * 1024      # (its weights are not bound yet)
    lin.bind({"w": torch.zeros(64, 128, dtype=dtype)}, dtype, "cpu")
    assert reserve([Norm(), outer]) == plain + times * SplitGemm.SCRATCH_BYTES


@pytest.mark.parametrize("hidden, F, E, top, act, tile", [(2048, 1024, 256, 8, "silu_glu", 256), (2048, 512, 1024, 8, "relu_squared", 256),
                                                          (1024, 704, 32, 4, "silu_glu", 256), (1024, 704, 700, 1, "clamped_glu", 128)])
def test_the_reserve_counts_the_grouped_rows_of_routed_experts(hidden, F, E, top, act, tile):
    """Inputs, hidden rows and sums of every pair and of the rows that pad each expert to whole tiles; a wrapped part counts them too."""
    from scriptling_llm_lib_b200.parts.experts import RoutedExperts
    gated = dict(gate_names=[f"g{j}" for j in range(E)], limit=7.0 if act == "clamped_glu" else None) if act != "relu_squared" else {}
    part = RoutedExperts(hidden, F, E, top, 1, 1, 1.0, "r", "c", [f"u{j}" for j in range(E)], [f"d{j}" for j in range(E)], act=act, **gated)
    rows = 16384
    padded = -(-(rows * top + E * (tile - 1)) // tile) * tile
    assert part._tile_rows(rows * top) == tile
    assert part.scratch_bytes(rows) == padded * (6 * hidden + 2 * F) + 4 * rows * hidden
    part.w_up = torch.empty((1, 1, 1))                      # kept in 32-bit: the FMA kernels' buffers
    assert part.scratch_bytes(rows) == rows * top * (4 * F * (3 if gated else 1) + 4 * hidden)


@pytest.mark.parametrize("dtype, n_seqs, H, G, D, V, pages, want", [
    (torch.bfloat16, 1, 16, 4, 64, 128, 1, True), (torch.bfloat16, 255, 16, 4, 64, 128, 1, True), (torch.bfloat16, 256, 16, 4, 64, 128, 1, False),
    (torch.bfloat16, 256, 16, 4, 64, 128, 2, True), (torch.bfloat16, 64, 64, 1, 32, 64, 1, False), (torch.bfloat16, 64, 64, 1, 32, 64, 3, True),
    (torch.float32, 1, 16, 4, 64, 128, 1, False), (torch.float32, 1, 16, 4, 64, 128, 2, False), (torch.float32, 1, 16, 4, 64, 128, 3, True),
    (torch.float32, 256, 16, 4, 64, 128, 2, True), (torch.float32, 1, 16, 16, 192, 128, 1, True), (torch.float32, 1, 16, 16, 192, 128, 2, False),
    (torch.float32, 128, 16, 2, 128, 256, 2, True), (torch.float32, 127, 16, 2, 128, 256, 2, False)])
def test_short_contexts_of_unequal_widths_keep_a_block_a_row_and_head(dtype, n_seqs, H, G, D, V, pages, want):
    """Two heads a block from 129 columns on, else four; the line lies at 1,024 blocks."""
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    assert KernelSet.attn_decode_split_pays(dtype, n_seqs, H, G, D, V, pages) == want


@pytest.mark.parametrize("M, N, K, want", [(65, 8192, 64, True), (65, 8200, 64, False), (128, 32768, 112, False), (128, 32768, 120, True), (129, 32768, 64, True)])
def test_few_rows_by_many_columns_with_short_sums_keep_the_chains(M, N, K, want):
    from scriptling_llm_lib_b200.csrc.bindings import SplitGemm
    assert SplitGemm.takes(torch.empty((M, K), device="meta"), torch.empty((N, K), device="meta")) == want


def test_the_map_of_pairs_to_rows_has_a_name_of_its_own():
    """Rows used to be gathered by the inverse map, as many int32 as this one where nothing pads: a call by the old name must not pass."""
    assert hasattr(MixKernels, "moe_spread_rows") and not hasattr(MixKernels, "moe_gather_rows")
