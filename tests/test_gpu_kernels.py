"""Each kernel alone against the plain implementation's function for the same op, at sizes other
than any model's (odd widths, head widths in steps of 16, vocabularies that are no power of two)."""
import math

import numpy as np
import pytest
import torch

import plain_llama as plain
from helpers import rel_err
from scriptling_llm_lib_b200.csrc.bindings import SplitGemm

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]
TOL = {torch.float32: 2e-6, torch.bfloat16: 6e-3}      # one op deep: float rounding / one bfloat16 rounding


@pytest.fixture(scope="module")
def kernel_sets():
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    return {dt: KernelSet(dt) for dt in DTYPES}


def dev(t, dtype=None):
    t = torch.as_tensor(t)
    return (t.to(dtype) if dtype is not None else t).cuda().contiguous()


def f64(t):
    return t.detach().cpu().to(torch.float64)


def rand(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g) * scale


# --------------------------------------------------------------------------- embedding
@pytest.mark.parametrize("dtype", DTYPES)
def test_embed_rows(kernel_sets, dtype):
    ks = kernel_sets[dtype]
    table = dev(rand(37, 24, seed=1), dtype)
    ids = dev([5, 0, 36, 5, 17], torch.int32)
    out = torch.empty(5, 24, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ks.embed_rows(ids, table, out, err)
    assert torch.equal(out.cpu(), table.float().cpu()[ids.cpu().long()]) and int(err) == 0
    ks.embed_rows(dev([3, 37], torch.int32), table, out[:2], err)       # an id outside the table: flagged, zeros
    assert int(err) == 1 and float(out[1].abs().sum()) == 0.0


# --------------------------------------------------------------------------- norm
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d, eps, w32", [(40, 1e-5, False), (2048, 1e-6, True), (1000, 1e-3, False), (13000, 1e-5, True)])
def test_add_rmsnorm(kernel_sets, dtype, d, eps, w32):
    ks = kernel_sets[dtype]
    T = 7
    x = dev(rand(T, d, seed=2, scale=3.0))
    delta = dev(rand(T, d, seed=3), dtype)
    w = dev(1.0 + rand(d, seed=4, scale=0.1), torch.float32 if w32 else torch.bfloat16)
    y = torch.empty(T, d, dtype=dtype, device="cuda")
    want_sum = f64(x) + f64(delta)
    want = plain.rms_norm(want_sum, f64(w), eps)
    xs = x.clone()
    ks.add_rmsnorm(xs, delta, None, w, y, eps)
    assert rel_err(y.cpu().float(), want) < TOL[dtype]
    assert rel_err(xs.cpu(), want_sum) < 2e-7                          # the residual sum is kept in 32-bit
    # no addend: x untouched
    xs = x.clone()
    ks.add_rmsnorm(xs, None, None, w, y, eps)
    assert torch.equal(xs, x) and rel_err(y.cpu().float(), plain.rms_norm(f64(x), f64(w), eps)) < TOL[dtype]
    # chosen rows: x untouched, rows of y follow `rows`
    rows = dev([6, 0, 3], torch.int32)
    y3 = torch.empty(3, d, dtype=dtype, device="cuda")
    xs = x.clone()
    ks.add_rmsnorm(xs, delta, rows, w, y3, eps)
    assert torch.equal(xs, x) and rel_err(y3.cpu().float(), want[[6, 0, 3]]) < TOL[dtype]
    # partial sums in float32
    parts = dev(rand(3, T, d, seed=5))
    xs = x.clone()
    ks.add_rmsnorm(xs, parts, None, w, y, eps)
    want_p = f64(x) + f64(parts).sum(0)
    assert rel_err(xs.cpu(), want_p) < 5e-7 and rel_err(y.cpu().float(), plain.rms_norm(want_p, f64(w), eps)) < TOL[dtype]
    ks.add_rmsnorm(x.clone(), parts, rows, w, y3, eps)
    assert rel_err(y3.cpu().float(), plain.rms_norm(want_p, f64(w), eps)[[6, 0, 3]]) < TOL[dtype]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d, w32", [(128, False), (896, True), (2048, False), (2176, True), (4096, False), (2000, False)])
def test_add_rmsnorm_many_rows(kernel_sets, dtype, d, w32):
    """The many rows of a prompt step (512 or more: small blocks with four accesses in flight per
    thread), with and without an addend, at widths that are and are not multiples of 128."""
    ks = kernel_sets[dtype]
    T, eps = 517, 1e-5
    x = dev(rand(T, d, seed=2, scale=3.0))
    delta = dev(rand(T, d, seed=3), dtype)
    w = dev(1.0 + rand(d, seed=4, scale=0.1), torch.float32 if w32 else torch.bfloat16)
    y = torch.full((T, d), float("nan"), dtype=dtype, device="cuda")
    want_sum = f64(x) + f64(delta)
    xs = x.clone()
    ks.add_rmsnorm(xs, delta, None, w, y, eps)
    assert rel_err(y.cpu().float(), plain.rms_norm(want_sum, f64(w), eps)) < TOL[dtype]
    assert rel_err(xs.cpu(), want_sum) < 2e-7
    xs = x.clone()
    y.fill_(float("nan"))
    ks.add_rmsnorm(xs, None, None, w, y, eps)
    assert torch.equal(xs, x) and rel_err(y.cpu().float(), plain.rms_norm(f64(x), f64(w), eps)) < TOL[dtype]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d", [512, 516, 2000, 2052, 8192, 16384])
def test_add_rmsnorm_many_rows_of_any_width(kernel_sets, dtype, d):
    """Rows in registers: widths that fill no access, partial sums as the addend, and rows picked out of the stream, which stays."""
    ks, T, eps = kernel_sets[dtype], 600, 1e-5
    x, w = dev(rand(T, d, seed=1, scale=2.0)), dev(rand(d, seed=3) + 1.0, dtype)
    parts = dev(rand(3, T, d, seed=4))
    y, xs = torch.full((T, d), float("nan"), dtype=dtype, device="cuda"), x.clone()
    ks.add_rmsnorm(xs, parts, None, w, y, eps)
    want = f64(x) + f64(parts).sum(0)
    assert rel_err(xs.cpu(), want) < 4e-7 and rel_err(y.cpu().float(), plain.rms_norm(want, f64(w), eps)) < TOL[dtype]
    rows, xs = dev(torch.arange(T - 1, -1, -1, dtype=torch.int32)), x.clone()
    ks.add_rmsnorm(xs, parts[:1], rows, w, y, eps)
    assert torch.equal(xs, x) and rel_err(y.cpu().float(), plain.rms_norm((f64(x) + f64(parts[0])).flip(0), f64(w), eps)) < TOL[dtype]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d", [12032, 12256, 12257, 12288, 12292])
def test_norms_of_rows_that_nearly_fill_what_a_block_may_have_unasked(kernel_sets, dtype, d):
    """A row of 12,288 floats is 48 KB, and the kernel has some shared memory of its own besides."""
    ks, T = kernel_sets[dtype], 3
    x, w = dev(rand(T, d, seed=1)), dev(rand(d, seed=3) + 1.0, dtype)
    y = torch.full((T, d), float("nan"), dtype=dtype, device="cuda")
    ks.add_rmsnorm(x, None, None, w, y, 1e-5)
    assert rel_err(y.cpu().float(), plain.rms_norm(f64(x), f64(w), 1e-5)) < TOL[dtype]
    y.fill_(float("nan"))
    ks.seq.add_norm(x, [], None, w, y, 1e-5, center=False)
    assert rel_err(y.cpu().float(), plain.rms_norm(f64(x), f64(w), 1e-5)) < TOL[dtype]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("dv", [4, 100, 127, 128, 132])
def test_unit_norms_of_heads(kernel_sets, dtype, dv):
    """The gated norm behind the delta rule and the unit keys and queries in front of it: heads of up to 128 by four elements, others."""
    seq, T, H, G = kernel_sets[dtype].seq, 37, 5, 3
    o, gate, w = dev(rand(T, H, dv, seed=1)), dev(rand(T, 8 + H * dv, seed=2), dtype), dev(rand(dv, seed=3) + 1.0, dtype)
    y = torch.full((T, H * dv), float("nan"), dtype=dtype, device="cuda")
    g = gate[:, 8:] if dtype == torch.bfloat16 or dv != 127 else gate[:, 7:7 + H * dv]
    seq.gated_unit_rms(o.view(T, H * dv), g, w, y, H, dv, 1e-6)
    od, gd = f64(o), f64(g.reshape(T, H, dv))
    want = od / torch.sqrt(od.square().mean(-1, keepdim=True) + 1e-6) * f64(w) * gd * torch.sigmoid(gd)
    assert rel_err(y.cpu().float(), want.reshape(T, H * dv)) < TOL[dtype]
    qk, ba, a_log, bias = dev(rand(T, 2 * G * dv, seed=5)), dev(rand(T, 2 * H, seed=6)), dev(rand(H, seed=7)), dev(rand(H, seed=8))
    bd, before = torch.full((T, 2 * H + G), float("nan"), device="cuda"), f64(qk).view(T, 2, G, dv)
    seq.delta_prepare(qk, ba, a_log, bias, bd, H, G, dv)
    unit = before / torch.sqrt(before.square().sum(-1, keepdim=True) + 1e-6)
    unit[:, 0] *= dv ** -0.5
    assert rel_err(qk.cpu(), unit.reshape(T, -1)) < 2e-6 and rel_err(bd[:, 2 * H:].cpu(), (unit[:, 0] * unit[:, 1]).sum(-1)) < 4e-6



# --------------------------------------------------------------------------- matrix products
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M, N, K", [(1, 33, 19), (3, 100, 72), (8, 64, 1000), (9, 130, 65), (70, 257, 136), (200, 96, 520),
                                     # K in multiples of 4: the 16-byte kernels (a block per four columns up to 8
                                     # rows, 64- and 128-row register tiles beyond), ragged edges everywhere
                                     (1, 35, 20), (2, 1003, 2048), (4, 6, 4100), (7, 515, 264), (9, 130, 64), (64, 300, 2048),
                                     (65, 129, 136), (300, 515, 264), (130, 1000, 24)])
def test_gemm_nt_generic(kernel_sets, dtype, M, N, K):
    ks = kernel_sets[dtype]
    a, w = dev(rand(M, K, seed=6), dtype), dev(rand(N, K, seed=7, scale=0.1), dtype)
    want = plain.linear(f64(a), f64(w))
    out = torch.empty(M, N, dtype=dtype, device="cuda")
    ks.gemm_nt(a, w, out)
    # float accumulation, float output: one ascending chain of K fused multiply-adds per output, whose
    # rounding error grows like sqrt(K) (2e-6 holds up to about a thousand terms)
    tol32 = 2e-6 * max(1.0, math.sqrt(K / 1024))
    if dtype == torch.float32:
        assert rel_err(out.cpu().float(), want) < tol32
    else:
        assert rel_err(out.cpu().float(), want) < TOL[dtype]
    out32 = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    ks.gemm_nt(a, w, out32)
    assert rel_err(out32.cpu(), want) < tol32
    if K % 4 == 0:
        for split in (2, 5):                                            # K cut into parts, partial sums for the reader
            parts = torch.full((split, M, N), float("nan"), dtype=torch.float32, device="cuda")
            ks.gemm_nt(a, w, parts)
            assert rel_err(parts.sum(0).cpu(), want) < tol32


def test_gemm_nt_generic_kernel_choice(kernel_sets):
    """One row of tiles on no more blocks than SMs keeps the kernel with a multiply-add an instruction."""
    for M, N, ksplit, pairs in [(65, 16384, 1, False), (128, 148 * 128, 1, False), (128, 148 * 128 + 1, 1, True), (96, 2048, 8, False),
                                (96, 6144, 6, True), (129, 128, 1, True), (2778, 1024, 1, True)]:
        assert all(bool(ks._fn("gemm_nt_pairs")(M, N, ksplit)) == pairs for ks in kernel_sets.values()), (M, N, ksplit)


def test_gemm_nt_generic_split_choice():
    from scriptling_llm_lib_b200.csrc.bindings import KernelSet
    assert KernelSet.gemm_nt_split(8, 2048, 8192, 148) == 1             # few rows: no cut
    assert KernelSet.gemm_nt_split(64, 2048, 8192, 148) == 16           # 16 tiles on 148 SMs: cut K
    assert KernelSet.gemm_nt_split(64, 2048, 2048, 148) == 8
    assert KernelSet.gemm_nt_split(2048, 8192, 2048, 148) == 1          # enough tiles
    assert KernelSet.gemm_nt_split(20, 96, 200, 148) == 1               # too shallow to cut


def test_attention_split_choice(kernel_sets):
    """About as many blocks as are resident at once (seven per SM for the one-head kernel, two or four
    for the grouped-query one), a tenth more at most, never more splits than pages, none without a page."""
    dk = kernel_sets[torch.bfloat16].decode
    one_head = {b: dk.attention_splits(b, 32, 32, 64, 64, 148) for b in (3, 4, 6, 8, 12, 16, 32, 64)}
    assert one_head == {3: 11, 4: 8, 6: 6, 8: 4, 12: 3, 16: 2, 32: 1, 64: 1}
    for b, n in one_head.items():
        assert n * 32 * b <= 1.12 * 7 * 148 or n == 1
    assert dk.attention_splits(8, 32, 32, 64, 3, 148) == 3                 # never more than pages
    assert dk.attention_splits(4, 32, 32, 64, 64, 148) * -(-64 // 8) == 64  # 9 were wanted: the ninth would be empty
    assert dk.attention_splits(8, 32, 8, 128, 64, 148) == 4                # grouped queries, width 128: two blocks per SM
    assert dk.attention_splits(8, 32, 8, 64, 64, 148) == 8                 # width 64: four (9 wanted, 8 pages each: 8)
    assert dk.attention_splits(8, 32, 8, 128, 8, 148) == 2                 # at least four pages each
    assert dk.attention_splits(1, 32, 32, 64, 64, 148) == 16               # a single sequence: the tensor-core kernel
    assert dk.attention_splits(500, 32, 32, 64, 64, 148) == 1


@pytest.mark.parametrize("M, N, K", [(1, 64, 64), (3, 100, 72), (8, 176, 64), (9, 1003, 144), (16, 2048, 2048),
                                     (33, 96, 200), (64, 640, 4096), (5, 49152 + 16, 256), (12, 16384, 128)])
def test_gemm_small_m(kernel_sets, M, N, K):
    """(The last two sizes, and the K splits of (16, 2048, 2048), have more blocks than are resident at once:
    they take the forms of the kernel with more blocks to an SM.)"""
    dk = kernel_sets[torch.bfloat16].decode
    a, w = dev(rand(M, K, seed=8), torch.bfloat16), dev(rand(N, K, seed=9, scale=0.05), torch.bfloat16)
    assert dk.takes(a, w)
    want = plain.linear(f64(a), f64(w))
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    dk.gemm_small_m(a, w, out)
    assert rel_err(out.cpu().float(), want) < TOL[torch.bfloat16]
    out32 = torch.empty(M, N, dtype=torch.float32, device="cuda")
    dk.gemm_small_m(a, w, out32)
    assert rel_err(out32.cpu(), want) < 3e-6
    for split in (2, 5):
        if K // split >= 8:
            parts = torch.full((split, M, N), float("nan"), dtype=torch.float32, device="cuda")
            dk.gemm_small_m(a, w, parts)
            assert rel_err(parts.sum(0).cpu(), want) < 3e-6
    if N % 16 == 0:
        F = N // 2
        tiled = w.view(2, F // 8, 8, K).permute(1, 0, 2, 3).reshape(N, K).contiguous()
        h = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
        dk.gemm_small_m(a, tiled, h, swiglu=True)
        assert rel_err(h.cpu().float(), plain.swiglu(want[:, :F], want[:, F:])) < TOL[torch.bfloat16]


@pytest.mark.parametrize("M, N, K, eps", [(1, 64, 64, 1e-5), (3, 112, 72, 1e-6), (8, 2048, 8192, 1e-5), (13, 1008, 144, 1e-3),
                                          (16, 2048, 2048, 1e-5), (5, 4096, 4104, 1e-5)])
def test_gemm_small_m_takes_over_the_halves_of_a_norm(kernel_sets, M, N, K, eps):
    """A norm folded into the products around it: the product before it adds to the residual stream,
    writes (residual * weight) in bfloat16 and leaves each tile's sums of squares; the product behind
    it scales its output rows by rsqrt(sum / width + eps). Both against the plain formulas, and the
    pair against the plain norm between two plain products."""
    dk = kernel_sets[torch.bfloat16].decode
    a, w = dev(rand(M, K, seed=8), torch.bfloat16), dev(rand(N, K, seed=9, scale=0.05), torch.bfloat16)
    resid0 = rand(M, N, seed=10, scale=2.0).float()
    norm_w = (1.0 + 0.1 * rand(N, seed=11)).float()
    y = plain.linear(f64(a), f64(w))
    # ---- the first half: residual += y, xb, sums of squares
    resid = dev(resid0, torch.float32)
    xb = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    sumsq = torch.full((-(-N // 16), M), float("nan"), dtype=torch.float32, device="cuda")
    dk.gemm_small_m(a, w, resid, fold=(dev(norm_w, torch.float32), xb, sumsq))
    want_resid = resid0.double() + y
    assert rel_err(resid.cpu(), want_resid) < 3e-6
    assert rel_err(xb.cpu().float(), want_resid * norm_w.double()) < TOL[torch.bfloat16]
    assert rel_err(sumsq.sum(0).cpu(), (want_resid ** 2).sum(1)) < 1e-5
    # ---- the second half: a product whose input rows are owed their scale
    w2 = dev(rand(48, N, seed=12, scale=0.05), torch.bfloat16)
    out = torch.empty(M, 48, dtype=torch.bfloat16, device="cuda")
    dk.gemm_small_m(xb, w2, out, owed=(sumsq, N, eps))
    scale = torch.rsqrt((resid.cpu().double() ** 2).mean(1) + eps)
    assert rel_err(out.cpu().float(), plain.linear(f64(xb), f64(w2)) * scale[:, None]) < TOL[torch.bfloat16]
    # ---- the pair is the plain norm between two plain products, up to where bfloat16 rounds
    normed = plain.rms_norm(want_resid, norm_w.double(), eps)
    assert rel_err(out.cpu().float(), plain.linear(normed, f64(w2))) < 2 * TOL[torch.bfloat16]
    # ---- the gated epilogue takes the scale too
    tiled = w2.view(2, 3, 8, N).permute(1, 0, 2, 3).reshape(48, N).contiguous()
    h = torch.empty(M, 24, dtype=torch.bfloat16, device="cuda")
    dk.gemm_small_m(xb, tiled, h, swiglu=True, owed=(sumsq, N, eps))
    full = plain.linear(f64(xb), f64(w2)) * scale[:, None]
    assert rel_err(h.cpu().float(), plain.swiglu(full[:, :24], full[:, 24:])) < TOL[torch.bfloat16]


@pytest.mark.parametrize("M, N, K, eps", [(130, 2048, 2048, 1e-5), (300, 1056, 520, 1e-6), (2048, 2048, 8192, 1e-5), (129, 160, 264, 1e-3),
                                          (700, 4096, 1024, 1e-5)])
def test_gemm_tc_takes_over_the_halves_of_a_norm(kernel_sets, M, N, K, eps):
    """The same two halves in the tensor-core products of a long prompt step: the residual sum,
    residual * weight and the sums of squares per 128 columns in the epilogue of one (staged through
    shared memory so that the float stream is read and written in whole rows); the row scale in the
    plain and the gated epilogue of the other, on the two-SM and the one-SM tiles."""
    tc = kernel_sets[torch.bfloat16].tensor_core
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w = dev(rand(M, K, seed=8), torch.bfloat16), dev(rand(N, K, seed=9, scale=0.05), torch.bfloat16)
    resid0 = rand(M, N, seed=10, scale=2.0).float()
    norm_w = (1.0 + 0.1 * rand(N, seed=11)).float()
    y = plain.linear(f64(a), f64(w))
    resid = dev(resid0, torch.float32)
    xb = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    sumsq = torch.full((-(-N // 128), M), float("nan"), dtype=torch.float32, device="cuda")
    tc.gemm(a, w, resid, err, fold=(dev(norm_w, torch.float32), xb, sumsq))
    want_resid = resid0.double() + y
    assert int(err) == 0
    assert rel_err(resid.cpu(), want_resid) < 3e-5             # tensor-core accumulation over long K, as in the plain product
    assert rel_err(xb.cpu().float(), want_resid * norm_w.double()) < TOL[torch.bfloat16]
    assert rel_err(sumsq.sum(0).cpu(), (want_resid ** 2).sum(1)) < 6e-5
    # the second half: plain and gated epilogues (48 columns: the one-SM tile)
    w2 = dev(rand(48, N, seed=12, scale=0.05), torch.bfloat16)
    scale = torch.rsqrt((resid.cpu().double() ** 2).mean(1) + eps)
    full = plain.linear(f64(xb), f64(w2)) * scale[:, None]
    out = torch.empty(M, 48, dtype=torch.bfloat16, device="cuda")
    tc.gemm(xb, w2, out, err, owed=(sumsq, N, eps))
    assert rel_err(out.cpu().float(), full) < TOL[torch.bfloat16]
    assert rel_err(out.cpu().float(), plain.linear(plain.rms_norm(want_resid, norm_w.double(), eps), f64(w2))) < 2 * TOL[torch.bfloat16]
    tiled = w2.view(2, 3, 8, N).permute(1, 0, 2, 3).reshape(48, N).contiguous()
    h = torch.empty(M, 24, dtype=torch.bfloat16, device="cuda")
    tc.gemm(xb, tiled, h, err, swiglu=True, owed=(sumsq, N, eps))
    assert rel_err(h.cpu().float(), plain.swiglu(full[:, :24], full[:, 24:])) < TOL[torch.bfloat16]
    # a wide product (the two-SM tile): every column tile of a row takes the same scale
    w3 = dev(rand(520, N, seed=13, scale=0.05), torch.bfloat16)
    out3 = torch.empty(M, 520, dtype=torch.float32, device="cuda")
    tc.gemm(xb, w3, out3, err, owed=(sumsq, N, eps))
    assert rel_err(out3.cpu(), plain.linear(f64(xb), f64(w3)) * scale[:, None]) < 3e-5
    assert int(err) == 0


@pytest.mark.parametrize("M, N, K", [(128, 128, 64), (100, 200, 72), (130, 264, 520), (2048, 2048, 2048), (65, 1003 * 8, 136),
                                     (300, 96, 8192), (257, 384, 136), (2304, 6400, 192), (1100, 4104, 2176)])
def test_gemm_tensor_core(kernel_sets, M, N, K):
    """The tcgen05 GEMM: bfloat16 and float outputs, the SiLU-gate epilogue.
    More than 128 rows and columns go to the kernel that pairs two SMs on a 256 x 256 tile: sizes with
    a ragged last tile, with several tiles to a pair (both accumulators, both phases), and with few
    and many k-blocks to a tile (eight or four epilogue warps)."""
    tc = kernel_sets[torch.bfloat16].tensor_core
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w = dev(rand(M, K, seed=14), torch.bfloat16), dev(rand(N, K, seed=15, scale=0.05), torch.bfloat16)
    assert tc.takes(a, w)
    want = plain.linear(f64(a), f64(w))
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    tc.gemm(a, w, out, err)
    assert rel_err(out.cpu().float(), want) < TOL[torch.bfloat16]
    out32 = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    tc.gemm(a, w, out32, err)
    assert rel_err(out32.cpu(), want) < 3e-5              # tensor-core accumulation over long K
    if N % 16 == 0:
        F = N // 2
        tiled = w.view(2, F // 8, 8, K).permute(1, 0, 2, 3).reshape(N, K).contiguous()
        h = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device="cuda")
        tc.gemm(a, tiled, h, err, swiglu=True)
        assert rel_err(h.cpu().float(), plain.swiglu(want[:, :F], want[:, F:])) < TOL[torch.bfloat16]
    assert int(err) == 0


@pytest.mark.parametrize("M, N, K", [(1, 128, 64), (17, 200, 72), (33, 264, 520), (64, 2048, 2048), (100, 1003 * 8, 136),
                                     (128, 96, 8192), (16, 6144, 2048)])
def test_gemm_tensor_core_few_rows(kernel_sets, M, N, K):
    """The weight-stationary tcgen05 GEMM for at most 128 rows: bfloat16 and float outputs, float partial
    sums of a split K (with more splits than some sizes have k-blocks to give), the SiLU-gate epilogue."""
    tc = kernel_sets[torch.bfloat16].tensor_core
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w = dev(rand(M, K, seed=24), torch.bfloat16), dev(rand(N, K, seed=25, scale=0.05), torch.bfloat16)
    want = plain.linear(f64(a), f64(w))
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    tc.gemm_skinny(a, w, out, err)
    assert rel_err(out.cpu().float(), want) < TOL[torch.bfloat16]
    out32 = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    tc.gemm_skinny(a, w, out32, err)
    assert rel_err(out32.cpu(), want) < 3e-5
    nkb = -(-K // 64)
    for split in sorted({min(2, nkb), min(4, nkb), min(7, nkb)} - {1}):
        parts = torch.full((split, M, N), float("nan"), dtype=torch.float32, device="cuda")
        tc.gemm_skinny(a, w, parts, err)
        assert rel_err(parts.cpu().double().sum(0), want) < 3e-5
    if N % 16 == 0:
        F = N // 2
        tiled = w.view(2, F // 8, 8, K).permute(1, 0, 2, 3).reshape(N, K).contiguous()
        h = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device="cuda")
        tc.gemm_skinny(a, tiled, h, err, swiglu=True)
        assert rel_err(h.cpu().float(), plain.swiglu(want[:, :F], want[:, F:])) < TOL[torch.bfloat16]
    assert int(err) == 0


@pytest.mark.parametrize("H, G, hd, rot, pairing", [(4, 2, 64, 64, "half"), (3, 1, 128, 128, "half"), (5, 5, 64, 24, "interleaved"),
                                                    (2, 1, 128, 128, "interleaved")])
def test_gemm_qkv_with_rotation_and_cache_write(kernel_sets, H, G, hd, rot, pairing):
    """The q|k|v product whose epilogue rotates queries and keys and puts keys and values into the pages:
    against product, rounding, rotation in plain float64; rows of two sequences at scattered positions."""
    from scriptling_llm_lib_b200.parts.rotary import RotaryEncoding
    tc = kernel_sets[torch.bfloat16].tensor_core
    enc = RotaryEncoding(hd, rot, 54321.0, None, pairing)
    enc.prepare(1024, "cuda")
    table, r, inter = enc.rotation()
    lens, pos0 = [150, 70], [60, 300]
    T, K, N = sum(lens), 136, (H + 2 * G) * hd
    a, w = dev(rand(T, K, seed=41), torch.bfloat16), dev(rand(N, K, seed=42, scale=0.1), torch.bfloat16)
    raw = plain.linear(f64(a), f64(w)).to(torch.bfloat16).to(torch.float64)          # the product, stored in bfloat16
    inv = plain.rope_inv_freq(rot, 54321.0)
    tok_pos = torch.cat([torch.arange(p, p + n) for n, p in zip(lens, pos0)])
    tok_seq = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)])
    q_want = plain.apply_rope(raw[:, :H * hd].view(T, H, hd), tok_pos, inv, pairing).reshape(T, H * hd)
    k_want = plain.apply_rope(raw[:, H * hd:(H + G) * hd].view(T, G, hd), tok_pos, inv, pairing)
    v_want = raw[:, (H + G) * hd:].view(T, G, hd)
    nan = lambda n: torch.full((n, G, hd), float("nan"))
    kp, vp, bt = paged([nan(p + n) for n, p in zip(lens, pos0)], [nan(p + n) for n, p in zip(lens, pos0)],
                       [p + n for n, p in zip(lens, pos0)], dtype=torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    qkv = torch.full((T, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    tc.gemm_qkv_rope(a, w, qkv, err, dev(tok_pos, torch.int32), dev(tok_seq, torch.int32), bt, table, kp, vp, H, G, hd, r, inter)
    assert int(err) == 0
    assert rel_err(qkv.cpu().float(), q_want) < TOL[torch.bfloat16]
    row = 0
    for b, (n, p) in enumerate(zip(lens, pos0)):
        for t in (0, 1, n // 2, n - 1):
            pos = p + t
            pg = int(bt[b, pos // PAGE])
            assert rel_err(f64(kp[pg, :, pos % PAGE]), k_want[row + t]) < TOL[torch.bfloat16]
            assert rel_err(f64(vp[pg, :, pos % PAGE]), v_want[row + t]) < 1e-6
        assert torch.isnan(kp[int(bt[b, 0]), :, 0].float()).all() if p > 0 else True     # places before the step untouched
        row += n


def test_gemm_small_m_refuses_what_it_cannot_take(kernel_sets):
    from scriptling_llm_lib_b200.csrc.bindings import KernelError
    dk = kernel_sets[torch.bfloat16].decode
    a, w = dev(rand(4, 36), torch.bfloat16), dev(rand(16, 36), torch.bfloat16)     # K no multiple of 8
    assert not dk.takes(a, w)
    with pytest.raises(KernelError):
        dk.gemm_small_m(a, w, torch.empty(4, 16, dtype=torch.bfloat16, device="cuda"))
    assert not dk.takes(dev(rand(65, 64), torch.bfloat16), dev(rand(16, 64), torch.bfloat16))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("F, tiled", [(176, True), (50, False), (8, True)])
def test_swiglu(kernel_sets, dtype, F, tiled):
    ks = kernel_sets[dtype]
    T = 5
    g, u = rand(T, F, seed=10, scale=2.0), rand(T, F, seed=11)
    gu = torch.cat([g, u], dim=1)
    if tiled:
        gu = torch.stack([g.view(T, F // 8, 8), u.view(T, F // 8, 8)], dim=2).reshape(T, 2 * F)
    gu = dev(gu, dtype)
    h = torch.empty(T, F, dtype=dtype, device="cuda")
    ks.swiglu(gu, h, tiled=tiled)
    gq, uq = f64(dev(g, dtype)), f64(dev(u, dtype))
    assert rel_err(h.cpu().float(), plain.swiglu(gq, uq)) < TOL[dtype]


# --------------------------------------------------------------------------- paged cache helpers
PAGE = 64


def paged(k, v, lengths, n_extra=3, seed=0, dtype=torch.float32):
    """Scatter per-sequence dense K/V [len, G, hd] into pages handed out in a scrambled order.
    Unused cache memory is NaN: a kernel that reads past a sequence's length shows it."""
    G, hd = k[0].shape[1], k[0].shape[2]
    need = [-(-n // PAGE) for n in lengths]
    total = sum(need) + n_extra
    order = np.random.default_rng(seed).permutation(total).tolist()
    kp = torch.full((total, G, PAGE, hd), float("nan"), dtype=torch.float32)
    vp = torch.full((total, G, PAGE, hd), float("nan"), dtype=torch.float32)
    bt = torch.full((len(lengths), max(need)), -1, dtype=torch.int32)
    for b, n in enumerate(lengths):
        for i in range(need[b]):
            pg = order.pop()
            bt[b, i] = pg
            m = min(PAGE, n - i * PAGE)
            kp[pg, :, :m] = k[b][i * PAGE:i * PAGE + m].permute(1, 0, 2)
            vp[pg, :, :m] = v[b][i * PAGE:i * PAGE + m].permute(1, 0, 2)
    return dev(kp, dtype), dev(vp, dtype), dev(bt)


@pytest.mark.parametrize("blocks, M, N, K", [(5, 130, 512, 256), (3, 65, 20, 12), (2, 128, 7, 100), (10, 300, 130, 64)])
def test_gemm_nt_blocks_is_every_block_by_itself(kernel_sets, blocks, M, N, K):
    """One launch for a block-diagonal product, on a column slice: the same bits as a launch a block (each output is one chain of
    multiply-adds in either)."""
    ks = kernel_sets[torch.float32]
    wide, w = dev(rand(M, blocks * K + 8, seed=3)), dev(rand(blocks, N, K, seed=4))
    a = wide[:, 4:4 + blocks * K]
    assert ks.gemm_nt_blocks_take(a, w) and not ks.gemm_nt_blocks_take(a[:64], w) and not ks.gemm_nt_blocks_take(wide[:, 1:1 + blocks * K], w)
    assert not ks.gemm_nt_blocks_take(a, torch.empty(w.numel() + 1, dtype=w.dtype, device="cuda")[1:].view(w.shape))
    out, each = (torch.full((blocks, M, N), float("nan"), device="cuda") for _ in range(2))
    ks.gemm_nt_blocks(a, w, out)
    for b in range(blocks):
        ks.gemm_nt(a[:, b * K:(b + 1) * K], w[b], each[b])
    assert torch.equal(out, each)
    want = torch.einsum("mbk,bnk->bmn", f64(a).view(M, blocks, K), f64(w))
    assert rel_err(out.cpu(), want) < TOL[torch.float32] * max(1.0, (K / 64) ** 0.5)


@pytest.mark.parametrize("M, N, K, split", [(33, 1, 1024, 8), (64, 300, 1000, 8), (129, 17, 2048, 8), (130, 256, 1032, 8), (300, 515, 4096, 8),
                                            (1000, 1000, 1024, 4), (2048, 72, 2048, 8), (2048, 576, 2048, 2), (300, 4096, 128, 1), (512, 2560, 1024, 1)])
def test_few_tiles_share_their_k_among_a_cluster(kernel_sets, M, N, K, split):
    """Products of a handful of tiles: ragged rows, columns, k-blocks and shares of them, both output types, rows of an odd stride, an
    activation on the sums; the sizes that stay with the kernels that walk all of K as well."""
    tc, flag = kernel_sets[torch.bfloat16].tensor_core, torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w = dev(rand(M, K + 8, seed=3), torch.bfloat16)[:, 8:], dev(rand(N, K, seed=4, scale=K ** -0.5), torch.bfloat16)
    assert tc.lib.sllm_gemm_tc_cluster_split(M, N, K, int(M <= 128)) == split
    run = tc.gemm_skinny if M <= 128 else tc.gemm
    want = f64(a) @ f64(w).T
    out32 = torch.full((M, N), float("nan"), device="cuda")
    run(a, w, out32, flag)
    assert rel_err(out32.cpu(), want) < 2e-5                             # sums in tensor memory, cut at every 16 terms
    wide = torch.full((M, N + 3), 7.0, dtype=torch.bfloat16, device="cuda")
    tc.gemm(a, w, wide[:, :N], flag)
    assert rel_err(wide[:, :N].cpu().float(), want) < TOL[torch.bfloat16] and bool((wide[:, N:] == 7.0).all())
    act = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    tc.gemm_act(a, w, act, flag, "relu_squared")
    assert rel_err(act.cpu().float(), want.clamp(min=0) ** 2) < TOL[torch.bfloat16] and int(flag) == 0


def test_a_product_of_what_the_kernel_in_front_writes(kernel_sets):
    """Both operands of a plain product may come out of the launch before it, also where a cluster shares its K."""
    tc, flag = kernel_sets[torch.bfloat16].tensor_core, torch.zeros(1, dtype=torch.int32, device="cuda")
    x, y, a = dev(rand(256, 8192, seed=1), torch.bfloat16), dev(rand(2048, 8192, seed=2, scale=8192 ** -0.5), torch.bfloat16), dev(rand(300, 2048, seed=3), torch.bfloat16)
    w, out, settled = (torch.zeros(s, device="cuda", dtype=t) for s, t in (((256, 2048), torch.bfloat16), ((300, 256), torch.float32), ((300, 256), torch.float32)))
    assert tc.lib.sllm_gemm_tc_cluster_split(300, 256, 2048, 0) > 1
    tc.gemm(x, y, w, flag)
    torch.cuda.synchronize()
    tc.gemm(a, w, settled, flag)
    for _ in range(5):
        w.zero_()
        tc.gemm(x, y, w, flag)
        tc.gemm(a, w, out, flag)
        assert torch.equal(out, settled) and int(flag) == 0


@pytest.mark.parametrize("M, N, K", [(17, 1, 128), (65, 7, 64), (128, 256, 72), (129, 129, 1000), (256, 128, 264), (257, 300, 4096), (700, 520, 136)])
def test_gemm_split_is_at_least_as_exact_as_the_chain(kernel_sets, M, N, K):
    """Products in three bfloat16 parts on the tensor cores: ragged tiles and k-blocks, K in parts (more than there are k-blocks among
    them), planes in portions. Sums end after 64 terms, so the error grows with sqrt(K / 64) from 2^-23, the terms left out and the
    last places cut within one sum; and it is no larger than that of the chains of multiply-adds."""
    ks = kernel_sets[torch.float32]
    wide, w = dev(rand(M, K + 8, seed=3)), dev(rand(N, K, seed=4))
    a, flag = wide[:, 4:4 + K], torch.zeros(1, dtype=torch.int32, device="cuda")
    want, tol = f64(a) @ f64(w).T, 2.0 ** -23 * (1 + 0.25 * math.sqrt(K / 64))
    off = lambda got: ((got.cpu().double() - want).norm() / want.norm()).item()                  # noqa: E731
    assert SplitGemm.takes(a, w) and not SplitGemm.takes(wide[:, 1:1 + K], w) and not SplitGemm.takes(a[:16], w)
    out, chain = (torch.full((M, N), float("nan"), device="cuda") for _ in range(2))
    ks.split.gemm(a, w, out, flag)
    ks.gemm_nt(a, w, chain)
    assert off(out) < min(tol, 1.05 * off(chain))
    for split in (2, 5):
        parts = torch.full((split, M, N), float("nan"), device="cuda")
        ks.split.gemm(a, w, parts, flag)
        assert off(parts.sum(0)) < 2 * tol
    class Portions(SplitGemm):
        SCRATCH_BYTES = 6 * K * 513                                      # 256 rows and columns at a time, or all of one of them
    again = torch.full((M, N), float("nan"), device="cuda")
    Portions().gemm(a, w, again, flag)
    assert torch.equal(again, out) and int(flag) == 0


@pytest.mark.parametrize("ea, ew, chained", [(-115, 0, False), (-125, 0, False), (0, -120, False), (-140, 20, False), (-100, 90, False),
                                             (100, -140, False), (-60, -50, False), (70, 40, True), (110, -60, True)])
def test_gemm_split_keeps_small_and_large_operands(kernel_sets, ea, ew, chained):
    """Operands as small as floats go, subnormal ones included, keep their 24 bits, also beside larger ones that meet a zero; what leaves the
    scaled range (operands above 2^104, sums from 2^80 on) comes out as the chain of multiply-adds has it."""
    ks, M, N, K = kernel_sets[torch.float32], 129, 40, 200
    a, w = dev(torch.ldexp(rand(M, K, seed=3), torch.tensor(ea))), dev(torch.ldexp(rand(N, K, seed=4), torch.tensor(ew)))
    a[:, 0], w[:, 0], w[:, 1], a[:, 1] = 1.0, 0.0, 1.0, 0.0
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    want, tol = f64(a) @ f64(w).T, 2.0 ** -23 * (1 + 0.25 * math.sqrt(K / 64))
    off = lambda got: ((got.cpu().double() - want).norm() / want.norm()).item()                  # noqa: E731
    out, chain = (torch.full((M, N), float("nan"), device="cuda") for _ in range(2))
    ks.split.gemm(a, w, out, flag)
    ks.gemm_nt(a, w, chain)
    assert int(flag) == 0 and (torch.equal(out[:, 1:], chain[:, 1:]) if chained else off(out) <= min(tol, 1.05 * off(chain)))


@pytest.mark.parametrize("M, N, K, parts", [(300, 200, 1032, 1), (300, 200, 1032, 3), (20, 129, 4096, 1), (6500, 12800, 64, 1)])
def test_gemm_split_sums_again_what_is_not_finite(kernel_sets, M, N, K, parts):
    """Rows, columns and single outputs that are not finite, in a block's first tiles and past its thirty-second, have the chain's values and
    the others keep theirs."""
    ks, flag = kernel_sets[torch.float32], torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w = dev(rand(M, K, seed=3)), dev(rand(N, K, seed=4))
    plain, out, chain = (torch.full((parts, M, N) if parts > 1 else (M, N), 7.0, device="cuda") for _ in range(3))
    ks.split.gemm(a, w, plain, flag)
    a[0], a[3, 1], a[M // 2, K - 1], a[M - 9:, 5], w[N - 1, 2] = math.nan, math.inf, -math.inf, 3.4e38, math.inf
    ks.split.gemm(a, w, out, flag)
    ks.gemm_nt(a, w, chain)
    bad = ~chain.isfinite()
    assert torch.equal(bad, ~out.isfinite()) and torch.equal(chain[bad].nan_to_num(1.5, 2.5, 3.5), out[bad].nan_to_num(1.5, 2.5, 3.5))
    touched = torch.zeros(M, N, dtype=torch.bool, device="cuda")
    touched[[0, 3, M // 2]], touched[M - 9:], touched[:, N - 1] = True, True, True
    assert torch.equal(out[..., ~touched], plain[..., ~touched]) and int(flag) == 0 and int(bad.sum()) >= parts * N
    assert rel_err(out[chain.abs() > 1e30].nan_to_num(0, 0, 0).cpu(), f64(chain[chain.abs() > 1e30].nan_to_num(0, 0, 0))) < 1e-6


def test_gemm_split_of_a_diverged_operand_is_no_hang(kernel_sets):
    """Every output not finite: a few times the chains' own kernel, and no wait near its limit. (An output a thread at a time took 100
    times as long.)"""
    ks, flag = kernel_sets[torch.float32], torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w, out = torch.full((1000, 2048), math.nan, device="cuda"), dev(rand(2560, 2048, seed=4)), torch.empty((1000, 2560), device="cuda")

    def us(run):
        run()
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        for _ in range(3):
            run()
        end.record()
        torch.cuda.synchronize()
        return start.elapsed_time(end) / 3

    assert us(lambda: ks.split.gemm(a, w, out, flag)) < 25 * us(lambda: ks.gemm_nt(a, w, out)) and bool(out.isnan().all()) and int(flag) == 0


def test_gemm_split_blocks_and_what_is_not_finite(kernel_sets):
    """A block-diagonal product in one launch; infinities, NaN and values whose first part rounds up to an infinity come out as the
    chain of multiply-adds has them."""
    ks, flag = kernel_sets[torch.float32], torch.zeros(1, dtype=torch.int32, device="cuda")
    blocks, M, N, K = 5, 300, 72, 72
    a, w = dev(rand(M, blocks * K, seed=3)), dev(rand(blocks, N, K, seed=4))
    for row, col, v in ((5, 3, math.inf), (7, 2, math.nan), (9, 1, 3.4e38), (11, 2 * K + 5, -math.inf)):
        a[row, col] = v
    w[1, 4, 6], w[3, 70, 71], a[12, K + 6] = -math.inf, 3.395e38, 0.0
    a[:, 4 * K - 1] = a[:, 4 * K - 1].clamp(-0.5, 0.5)                   # 3.395e38 times it stays finite
    out, chain = (torch.full((blocks, M, N), 7.0, device="cuda") for _ in range(2))
    ks.split.blocks(a, w, out, flag)
    ks.gemm_nt_blocks(a, w, chain)
    bad = ~chain.isfinite()
    assert bad.sum() > 4 * N and torch.equal(bad, ~out.isfinite()) and int(flag) == 0
    assert torch.equal(chain[bad].nan_to_num(1.5, 2.5, 3.5), out[bad].nan_to_num(1.5, 2.5, 3.5))
    large = chain.abs() > 1e30
    assert ((out - chain)[large & ~bad] / chain[large & ~bad]).abs().max() < 1e-6
    rest = ~(bad | large)
    assert rel_err(out[rest].cpu(), f64(chain[rest])) < 4e-7


# --------------------------------------------------------------------------- rotary + cache write
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H, G, hd, rot, pairing", [(4, 2, 16, 16, "interleaved"), (3, 1, 32, 16, "half"),
                                                    (6, 3, 48, 48, "half"), (2, 2, 80, 40, "interleaved"),
                                                    (2, 1, 16, 8, "half"), (5, 5, 32, 12, "interleaved")])
def test_rope_kv_write(kernel_sets, dtype, H, G, hd, rot, pairing):
    from scriptling_llm_lib_b200.parts.rotary import RotaryEncoding
    ks = kernel_sets[dtype]
    enc = RotaryEncoding(hd, rot, 12345.0, None, pairing)
    enc.prepare(300, "cuda")
    lens, pos0 = [5, 70, 1], [0, 60, 199]                               # new tokens and tokens already cached
    T = sum(lens)
    qkv = dev(rand(T, (H + 2 * G) * hd, seed=12), dtype)
    tok_seq = np.repeat(np.arange(3), lens)
    tok_pos = np.concatenate([np.arange(p, p + n) for p, n in zip(pos0, lens)])
    n_pages = 9
    kp = torch.zeros(n_pages, G, PAGE, hd, dtype=dtype, device="cuda")
    vp = torch.zeros_like(kp)
    bt = dev([[7, -1, -1, -1], [2, 5, 0, -1], [1, 3, 8, 4]], torch.int32)
    orig = f64(qkv).clone()
    ks.rope_kv_write(qkv, dev(tok_pos, torch.int32), dev(tok_seq, torch.int32), bt, enc.cos_sin, kp, vp, H, G, hd, rot,
                     pairing == "interleaved")
    inv = plain.rope_inv_freq(rot, 12345.0)
    pos_t = torch.as_tensor(tok_pos)
    q_want = plain.apply_rope(orig[:, :H * hd].view(T, H, hd), pos_t, inv, pairing)
    k_want = plain.apply_rope(orig[:, H * hd:(H + G) * hd].view(T, G, hd), pos_t, inv, pairing)
    v_want = orig[:, (H + G) * hd:].view(T, G, hd)
    assert rel_err(f64(qkv)[:, :H * hd], q_want.reshape(T, -1)) < TOL[dtype]
    assert torch.equal(f64(qkv)[:, H * hd:], orig[:, H * hd:])          # k and v columns of the buffer are not rewritten
    for t in range(T):
        pg = int(bt[tok_seq[t], tok_pos[t] // PAGE])
        assert rel_err(f64(kp[pg, :, tok_pos[t] % PAGE]), k_want[t]) < TOL[dtype]
        assert torch.equal(f64(vp[pg, :, tok_pos[t] % PAGE]), v_want[t])
    assert float(kp[6].abs().sum()) == 0.0                               # a page nobody owns stays untouched
    # queries only (a layer that reads another layer's cache)
    q2 = dev(rand(T, H * hd, seed=13), dtype)
    o2 = f64(q2).clone()
    ks.rope_kv_write(q2, dev(tok_pos, torch.int32), dev(tok_seq, torch.int32), bt, enc.cos_sin, None, None, H, 0, hd, rot,
                     pairing == "interleaved")
    assert rel_err(f64(q2), plain.apply_rope(o2.view(T, H, hd), pos_t, inv, pairing).reshape(T, -1)) < TOL[dtype]


# --------------------------------------------------------------------------- attention
def attention_case(H, G, hd, lens, pos0, seed):
    """Per sequence: all keys/values (cached + new) and the new queries."""
    ks_, vs_, qs_ = [], [], []
    for b, (n, p) in enumerate(zip(lens, pos0)):
        ks_.append(rand(p + n, G, hd, seed=seed + 3 * b))
        vs_.append(rand(p + n, G, hd, seed=seed + 3 * b + 1))
        qs_.append(rand(n, H, hd, seed=seed + 3 * b + 2, scale=2.0))
    return qs_, ks_, vs_


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H, G, hd, window", [(4, 2, 16, None), (3, 1, 32, None), (6, 3, 48, 24), (2, 2, 80, None),
                                              (8, 2, 64, 100), (2, 1, 128, None)])
def test_attn_paged(kernel_sets, dtype, H, G, hd, window):
    ks = kernel_sets[dtype]
    lens, pos0 = [37, 1, 130, 16], [0, 250, 70, 64]
    qs, kk, vv = attention_case(H, G, hd, lens, pos0, 20)
    rnd = (lambda t: t) if dtype == torch.float32 else (lambda t: t.bfloat16().float())
    qs, kk, vv = [rnd(t) for t in qs], [rnd(t) for t in kk], [rnd(t) for t in vv]
    kp, vp, bt = paged(kk, vv, [p + n for p, n in zip(pos0, lens)], dtype=dtype)
    T = sum(lens)
    q = dev(torch.cat([t.reshape(t.shape[0], -1) for t in qs]), dtype)
    out = torch.empty(T, H * hd, dtype=dtype, device="cuda")
    seq_start = dev(np.concatenate([[0], np.cumsum(lens)]), torch.int32)
    ks.attn_paged(q, out, seq_start, dev(pos0, torch.int32), bt, kp, vp, len(lens), max(lens), H, G, hd, window,
                  1.0 / math.sqrt(hd))
    want = torch.cat([plain.attention(f64(qs[b]), f64(kk[b]), f64(vv[b]), torch.arange(pos0[b], pos0[b] + lens[b]),
                                      torch.arange(pos0[b] + lens[b]), window).reshape(lens[b], -1) for b in range(len(lens))])
    # a score is a chain of head_dim float multiply-adds: its rounding, and with it the probabilities', grows
    # like sqrt(head_dim) (2e-6 holds up to a width of 64)
    assert rel_err(out.cpu().float(), want) < TOL[dtype] * (max(1.0, math.sqrt(hd / 64)) if dtype == torch.float32 else 1.0)
    # few new rows per sequence: the one-query-at-a-time form of the kernel
    lens2 = [3, 1, 2, 4]
    qs2 = [t[:n] for t, n in zip(qs, lens2)]
    kp2, vp2, bt2 = paged([k[:p + n] for k, p, n in zip(kk, pos0, lens2)], [v[:p + n] for v, p, n in zip(vv, pos0, lens2)],
                          [p + n for p, n in zip(pos0, lens2)], dtype=dtype, seed=5)
    q2 = dev(torch.cat([t.reshape(t.shape[0], -1) for t in qs2]), dtype)
    out2 = torch.empty(sum(lens2), H * hd, dtype=dtype, device="cuda")
    ks.attn_paged(q2, out2, dev(np.concatenate([[0], np.cumsum(lens2)]), torch.int32), dev(pos0, torch.int32), bt2, kp2, vp2,
                  len(lens2), max(lens2), H, G, hd, window, 1.0 / math.sqrt(hd))
    want2 = torch.cat([plain.attention(f64(qs2[b]), f64(kk[b][:pos0[b] + lens2[b]]), f64(vv[b][:pos0[b] + lens2[b]]),
                                       torch.arange(pos0[b], pos0[b] + lens2[b]), torch.arange(pos0[b] + lens2[b]),
                                       window).reshape(lens2[b], -1) for b in range(len(lens2))])
    assert rel_err(out2.cpu().float(), want2) < TOL[dtype] * (max(1.0, math.sqrt(hd / 64)) if dtype == torch.float32 else 1.0)


@pytest.mark.parametrize("lens, pos0", [([37, 1, 130, 64, 200, 128], [0, 250, 70, 64, 0, 300]), ([37], [0]), ([1], [700]),
                                        ([2, 3], [63, 64])])
@pytest.mark.parametrize("H, G, window", [(4, 2, None), (3, 1, None), (6, 3, 24), (8, 2, 100), (5, 5, 1), (2, 2, 64)])
@pytest.mark.parametrize("hd", [64, 128])
def test_attn_prefill_tcgen05(kernel_sets, hd, H, G, window, lens, pos0):
    """The tcgen05 attention (S and P V in tensor memory, TMA-fed pages), heads of 64 and of 128: prompts
    that start at a non-empty cache, a one-token prompt, tiles of exactly 64 and 128 queries, windows;
    unused cache memory is NaN, which the kernel must never let through."""
    fa = kernel_sets[torch.bfloat16].prefill_attention_tc
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    qs, kk, vv = attention_case(H, G, hd, lens, pos0, 30)
    rnd = lambda t: t.bfloat16().float()
    qs, kk, vv = [rnd(t) for t in qs], [rnd(t) for t in kk], [rnd(t) for t in vv]
    kp, vp, bt = paged(kk, vv, [p + n for p, n in zip(pos0, lens)], dtype=torch.bfloat16)
    T = sum(lens)
    q = dev(torch.cat([t.reshape(t.shape[0], -1) for t in qs]), torch.bfloat16)
    out = torch.full((T, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    seq_start = dev(np.concatenate([[0], np.cumsum(lens)]), torch.int32)
    fa.attn(q, out, seq_start, dev(pos0, torch.int32), bt, kp, vp, len(lens), max(lens), H, G, hd, window, 1.0 / math.sqrt(hd), err)
    want = torch.cat([plain.attention(f64(qs[b]), f64(kk[b]), f64(vv[b]), torch.arange(pos0[b], pos0[b] + lens[b]),
                                      torch.arange(pos0[b] + lens[b]), window).reshape(lens[b], -1) for b in range(len(lens))])
    assert int(err) == 0
    assert rel_err(out.cpu().float(), want) < 1.2e-2          # probabilities are rounded to bfloat16 before P V


@pytest.mark.parametrize("lens, pos0", [([37, 1, 130, 64, 200, 128], [0, 250, 70, 64, 0, 300]), ([1], [700]), ([700], [0]),
                                        ([300, 513, 1], [77, 0, 100])])
@pytest.mark.parametrize("kd, vd, H, G, window", [(64, 64, 4, 2, 0), (64, 128, 4, 1, 100), (128, 64, 3, 3, 0), (128, 128, 4, 4, -96),
                                                  (192, 128, 3, 3, 0), (192, 64, 4, 2, 65), (136, 72, 6, 3, 0), (8, 8, 2, 1, 0),
                                                  (80, 80, 2, 2, 1), (176, 120, 2, 1, 0)])
def test_attn_prefill_tcgen05_with_float_weights(kernel_sets, kd, vd, H, G, window, lens, pos0):
    """Softmax weights in three bfloat16 parts: what is left against 64 bits is the output's own rounding to 8 significant
    bits (at most 2^-8 of an element) and float sums far below it. Unused cache memory is NaN; windows and (below 0) chunks."""
    fa = kernel_sets[torch.bfloat16].prefill_attention_tc
    assert fa.takes(kd, vd, exact_weights=True) and not fa.takes(200, 64, exact_weights=True) and not fa.takes(192, 64)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rnd = lambda t: t.bfloat16().float()
    held = [p + n for p, n in zip(pos0, lens)]
    kk = [rnd(rand(n, G, kd, seed=50 + 3 * b)) for b, n in enumerate(held)]
    vv = [rnd(rand(n, G, vd, seed=51 + 3 * b)) for b, n in enumerate(held)]
    qs = [rnd(rand(n, H, kd, seed=52 + 3 * b, scale=3.0)) for b, n in enumerate(lens)]
    kp, _, bt = paged(kk, kk, held, dtype=torch.bfloat16)
    vp, _, _ = paged(vv, vv, held, dtype=torch.bfloat16)
    q = dev(torch.cat([t.reshape(t.shape[0], -1) for t in qs]), torch.bfloat16)
    out = torch.full((sum(lens), H * vd), float("nan"), dtype=torch.bfloat16, device="cuda")
    seq_start = dev(np.concatenate([[0], np.cumsum(lens)]), torch.int32)
    fa.attn(q, out, seq_start, dev(pos0, torch.int32), bt, kp, vp, len(lens), max(lens), H, G, kd, window, kd ** -0.5, err, v_dim=vd,
            exact_weights=True)
    want = []
    for b, (n, p) in enumerate(zip(lens, pos0)):
        at, key = torch.arange(p, p + n)[:, None], torch.arange(p + n)[None, :]
        first = torch.zeros_like(at) if window == 0 else at - window + 1 if window > 0 else at - at % -window
        k, v = (f64(t).repeat_interleave(H // G, 1) for t in (kk[b], vv[b]))
        sc = torch.einsum("qhd,khd->hqk", f64(qs[b]), k) * kd ** -0.5
        sc = sc.masked_fill((key > at) | (key < first), -math.inf).softmax(-1)
        want.append(torch.einsum("hqk,khd->qhd", sc, v).reshape(n, -1))
    assert int(err) == 0
    assert rel_err(out.cpu().float(), torch.cat(want)) < 2.0 ** -8 + 2e-5


@pytest.mark.parametrize("kd, vd, H, G, window", [(64, 128, 48, 6, 300), (192, 128, 40, 40, 0), (128, 64, 64, 8, -128)])
def test_attn_prefill_with_float_weights_many_items(kernel_sets, kd, vd, H, G, window):
    """More work items than blocks that stay: a block's rings, accumulators and maxima go on from one item to the next, among them items of
    one key tile and of two. Rows at the tiles' edges against 64 bits, to the output's rounding and float sums below it."""
    fa, err = kernel_sets[torch.bfloat16].prefill_attention_tc, torch.zeros(1, dtype=torch.int32, device="cuda")
    lens, pos0, g = [900, 40, 129], [0, 0, 500], torch.Generator().manual_seed(kd)
    draw = lambda *s: torch.randn(*s, generator=g).bfloat16().float()      # noqa: E731
    held = [p + n for p, n in zip(pos0, lens)]
    kk, vv, qs = [draw(n, G, kd) for n in held], [draw(n, G, vd) for n in held], [draw(n, H, kd) for n in lens]
    kp, _, bt = paged(kk, kk, held, dtype=torch.bfloat16)
    vp, _, _ = paged(vv, vv, held, dtype=torch.bfloat16)
    q, out = dev(torch.cat([t.reshape(t.shape[0], -1) for t in qs]), torch.bfloat16), torch.full((sum(lens), H * vd), 7.0, dtype=torch.bfloat16, device="cuda")
    fa.attn(q, out, dev(np.concatenate([[0], np.cumsum(lens)]), torch.int32), dev(pos0, torch.int32), bt, kp, vp, len(lens), max(lens), H, G, kd, window,
            kd ** -0.5, err, v_dim=vd, exact_weights=True)
    row0 = 0
    for b, (n, p) in enumerate(zip(lens, pos0)):
        rows = torch.tensor(sorted({0, 1, 39, 63, 64, 127, 128, 255, 256, 700, n - 1} & set(range(n))))
        at, key = (p + rows)[:, None], torch.arange(p + n)[None, :]
        first = torch.zeros_like(at) if window == 0 else at - window + 1 if window > 0 else at - at % -window
        k, v = (f64(t).repeat_interleave(H // G, 1) for t in (kk[b], vv[b]))
        sc = (torch.einsum("qhd,khd->hqk", f64(qs[b][rows]), k) * kd ** -0.5).masked_fill((key > at) | (key < first), -math.inf).softmax(-1)
        want = torch.einsum("hqk,khd->qhd", sc, v).reshape(len(rows), -1)
        assert rel_err(out[row0 + rows].cpu().float(), want) < 2.0 ** -8 + 2e-5
        row0 += n
    assert int(err) == 0


@pytest.mark.parametrize("hd, H, G, window", [(64, 40, 40, None), (64, 24, 6, 700), (128, 24, 6, None), (128, 15, 15, None), (128, 9, 3, 900)])
def test_attn_prefill_tcgen05_long_prompts_many_items(kernel_sets, hd, H, G, window):
    """Prompts of a few thousand tokens and more work items than resident blocks: every block walks several
    items, the key/value ring wraps many times, and at head width 128 both ways of pairing query tiles are
    taken (two heads of a group; two consecutive tiles of one head where the group is odd). Sampled rows
    (the first, the last, the edges of the 64- and 128-row tiles) against the plain implementation, every
    row against the generic kernel."""
    ks = kernel_sets[torch.bfloat16]
    fa = ks.prefill_attention_tc
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    lens, pos0 = [2100, 1500], [0, 64]
    g = torch.Generator().manual_seed(hd + H)
    rnd = lambda t: t.bfloat16().float()
    kk = [rnd(torch.randn(p + n, G, hd, generator=g)) for p, n in zip(pos0, lens)]
    vv = [rnd(torch.randn(p + n, G, hd, generator=g)) for p, n in zip(pos0, lens)]
    qs = [rnd(torch.randn(n, H, hd, generator=g)) for n in lens]
    kp, vp, bt = paged(kk, vv, [p + n for p, n in zip(pos0, lens)], dtype=torch.bfloat16)
    T = sum(lens)
    q = dev(torch.cat([t.reshape(t.shape[0], -1) for t in qs]), torch.bfloat16)
    seq_start = dev(np.concatenate([[0], np.cumsum(lens)]), torch.int32)
    out = torch.full((T, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    fa.attn(q, out, seq_start, dev(pos0, torch.int32), bt, kp, vp, len(lens), max(lens), H, G, hd, window, 1.0 / math.sqrt(hd), err)
    assert int(err) == 0
    got = out.cpu().float()
    assert torch.isfinite(got).all()
    row0 = 0
    for b, n in enumerate(lens):
        rows = sorted({0, 1, 62, 63, 64, 65, 126, 127, 128, 129, 191, 192, 255, 256, 1023, 1024, n - 129, n - 128, n - 65, n - 64, n - 2, n - 1}
                      | {int(x) for x in torch.randint(0, n, (24,), generator=g)})
        idx = torch.tensor(rows)
        want = plain.attention(f64(qs[b][idx]), f64(kk[b]), f64(vv[b]), pos0[b] + idx, torch.arange(pos0[b] + n), window).reshape(len(rows), -1)
        assert rel_err(got[row0 + idx], want) < 1.2e-2, (b, hd, H, G)
        row0 += n
    other = torch.empty_like(out)
    ks.attn_paged(q, other, seq_start, dev(pos0, torch.int32), bt, kp, vp, len(lens), max(lens), H, G, hd, window, 1.0 / math.sqrt(hd))
    assert rel_err(got, other.cpu().float()) < 1.5e-2


@pytest.mark.parametrize("hd, H, G", [(64, 32, 32), (128, 32, 8), (128, 5, 5)])
def test_attn_prefill_tcgen05_same_bits_every_launch(kernel_sets, hd, H, G):
    """The hand-overs between the kernel's roles must not let timing into the result: twenty launches on
    the same input, unequal prompts, give the same bits (a buffer reused a phase too early shows here)."""
    fa = kernel_sets[torch.bfloat16].prefill_attention_tc
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    lens = [1943, 560, 700, 65, 1, 1024]
    g = torch.Generator().manual_seed(hd + H)
    kk = [torch.randn(n, G, hd, generator=g) for n in lens]
    vv = [torch.randn(n, G, hd, generator=g) for n in lens]
    kp, vp, bt = paged(kk, vv, lens, dtype=torch.bfloat16)
    T = sum(lens)
    q = dev(torch.randn(T, H * hd, generator=g), torch.bfloat16)
    seq_start = dev(np.concatenate([[0], np.cumsum(lens)]), torch.int32)
    pos0 = dev([0] * len(lens), torch.int32)
    first = None
    for _ in range(20):
        out = torch.full((T, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
        fa.attn(q, out, seq_start, pos0, bt, kp, vp, len(lens), max(lens), H, G, hd, None, 1.0 / math.sqrt(hd), err)
        if first is None:
            first = out
            assert torch.isfinite(first.float()).all()
        else:
            assert torch.equal(out, first)
    assert int(err) == 0


@pytest.mark.parametrize("H, G, hd, window", [(4, 2, 16, None), (3, 1, 32, None), (32, 32, 64, None), (8, 2, 128, 300),
                                              (4, 1, 64, 65), (2, 2, 256, None),
                                              # two or more query heads per key/value head at widths 64 and 128: the
                                              # tensor-core variant; 12 and 40 heads per group use its upper rows and loop
                                              (32, 8, 64, None), (9, 3, 64, 100), (6, 3, 128, None), (24, 2, 64, 17),
                                              (40, 1, 128, 500),
                                              # one head per group, few (sequence, head) pairs: the same variant
                                              (4, 4, 64, None), (8, 8, 128, 70)])
@pytest.mark.parametrize("n_split", [1, 3, 16, 40, 70])      # 70: more than the merging block weighs in one pass
def test_attn_decode(kernel_sets, H, G, hd, window, n_split):
    dk = kernel_sets[torch.bfloat16].decode
    lens, pos0 = [1, 1, 1, 1, 1], [0, 63, 64, 700, 257]
    qs, kk, vv = attention_case(H, G, hd, lens, pos0, 40)
    rnd = lambda t: t.bfloat16().float()
    qs, kk, vv = [rnd(t) for t in qs], [rnd(t) for t in kk], [rnd(t) for t in vv]
    kp, vp, bt = paged(kk, vv, [p + 1 for p in pos0], dtype=torch.bfloat16)
    q = dev(torch.cat([t.reshape(1, -1) for t in qs]), torch.bfloat16)
    B = len(lens)
    out = torch.empty(B, H * hd, dtype=torch.bfloat16, device="cuda")
    scratch = torch.full((B * H * n_split * (hd + 2),), float("nan"), dtype=torch.float32, device="cuda")
    dk.attn_decode(q, out, dev(pos0, torch.int32), bt, kp, vp, scratch, B, H, G, hd, window, 1.0 / math.sqrt(hd), n_split)
    want = torch.cat([plain.attention(f64(qs[b]), f64(kk[b]), f64(vv[b]), torch.tensor([pos0[b]]),
                                      torch.arange(pos0[b] + 1), window).reshape(1, -1) for b in range(B)])
    assert rel_err(out.cpu().float(), want) < TOL[torch.bfloat16]
    # one kernel: the last split to finish merges; twice, the tickets must come back to zero
    tickets = torch.zeros(B * G, dtype=torch.int32, device="cuda")
    for _ in range(2):
        out.fill_(float("nan"))
        scratch.fill_(float("nan"))
        dk.attn_decode(q, out, dev(pos0, torch.int32), bt, kp, vp, scratch, B, H, G, hd, window, 1.0 / math.sqrt(hd), n_split,
                       tickets=tickets)
        assert rel_err(out.cpu().float(), want) < TOL[torch.bfloat16]
        assert int(tickets.abs().sum()) == 0


@pytest.mark.parametrize("H, G, hd, rot, pairing, window", [(4, 2, 16, 16, "half", None), (3, 1, 32, 16, "interleaved", None),
                                                            (32, 32, 64, 64, "half", None), (8, 2, 128, 64, "half", 300),
                                                            (4, 4, 64, 8, "interleaved", 65),
                                                            (9, 3, 64, 64, "half", 70), (12, 1, 64, 32, "interleaved", None),
                                                            (32, 8, 128, 128, "half", None)])
@pytest.mark.parametrize("n_split", [1, 5])
def test_attn_decode_with_rotation_and_cache_write_fused(kernel_sets, H, G, hd, rot, pairing, window, n_split):
    """One kernel does what rope_kv_write + attn_decode do: rotate q, rotate and store the new key,
    store the new value, attend. Checked against the plain functions, and the cache afterwards."""
    from scriptling_llm_lib_b200.parts.rotary import RotaryEncoding
    dk = kernel_sets[torch.bfloat16].decode
    enc = RotaryEncoding(hd, rot, 54321.0, None, pairing)
    enc.prepare(1024, "cuda")
    assert dk.rotation_fusable(rot, pairing == "interleaved")
    pos0 = [0, 63, 64, 700, 257]
    B = len(pos0)
    rnd = lambda t: t.bfloat16().float()
    old_k = [rnd(rand(p, G, hd, seed=90 + b)) for b, p in enumerate(pos0)]           # cached (already rotated) keys
    old_v = [rnd(rand(p, G, hd, seed=95 + b)) for b, p in enumerate(pos0)]
    raw = rnd(rand(B, (H + 2 * G) * hd, seed=99, scale=1.5))                         # this step's unrotated q | k | v
    inv = plain.rope_inv_freq(rot, 54321.0)
    q_rot, k_new, v_new = [], [], []
    for b, p in enumerate(pos0):
        pos = torch.tensor([p])
        q_rot.append(rnd(plain.apply_rope(f64(raw[b:b + 1, :H * hd]).view(1, H, hd), pos, inv, pairing).float()))
        k_new.append(rnd(plain.apply_rope(f64(raw[b:b + 1, H * hd:(H + G) * hd]).view(1, G, hd), pos, inv, pairing).float()))
        v_new.append(raw[b:b + 1, (H + G) * hd:].view(1, G, hd))
    want = torch.cat([plain.attention(f64(q_rot[b]), f64(torch.cat([old_k[b], k_new[b]])), f64(torch.cat([old_v[b], v_new[b]])),
                                      torch.tensor([pos0[b]]), torch.arange(pos0[b] + 1), window).reshape(1, -1) for b in range(B)])
    # pages sized for pos0 + 1 keys; the new key's place holds NaN until the kernel writes it
    nan_row = torch.full((1, G, hd), float("nan"))
    kp, vp, bt = paged([torch.cat([old_k[b], nan_row]) for b in range(B)], [torch.cat([old_v[b], nan_row]) for b in range(B)],
                       [p + 1 for p in pos0], dtype=torch.bfloat16)
    out = torch.full((B, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    scratch = torch.full((B * H * n_split * (hd + 2),), float("nan"), dtype=torch.float32, device="cuda")
    tickets = torch.zeros(B * G, dtype=torch.int32, device="cuda")
    dk.attn_decode_rope(dev(raw, torch.bfloat16), out, dev(pos0, torch.int32), bt, kp, vp, scratch, tickets, enc.cos_sin, rot,
                        pairing == "interleaved", True, B, H, G, hd, window, 1.0 / math.sqrt(hd), n_split)
    assert rel_err(out.cpu().float(), want) < TOL[torch.bfloat16]
    assert int(tickets.abs().sum()) == 0
    for b, p in enumerate(pos0):
        pg = int(bt[b, p // PAGE])
        assert rel_err(f64(kp[pg, :, p % PAGE]), f64(k_new[b][0])) < TOL[torch.bfloat16]
        assert torch.equal(f64(vp[pg, :, p % PAGE]), f64(v_new[b][0]))
    # a layer that reads another layer's cache: queries only, the key at the query's position is read, not written
    out2 = torch.full((B, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    dk.attn_decode_rope(dev(raw[:, :H * hd], torch.bfloat16), out2, dev(pos0, torch.int32), bt, kp, vp, scratch, tickets,
                        enc.cos_sin, rot, pairing == "interleaved", False, B, H, G, hd, window, 1.0 / math.sqrt(hd), n_split)
    assert rel_err(out2.cpu().float(), want) < TOL[torch.bfloat16]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H, G, hd, window", [(4, 2, 16, None), (3, 1, 32, 40), (6, 3, 48, None), (32, 32, 64, None),
                                              (2, 2, 80, 100), (8, 2, 128, 300), (2, 1, 256, None), (2, 2, 320, 65)])
@pytest.mark.parametrize("n_split", [1, 3, 16])
def test_attn_decode_split_generic(kernel_sets, dtype, H, G, hd, window, n_split):
    """The decode attention of the generic path (all of the 32-bit decode step): head widths in
    steps of 4 elements up to 512, any grouping, windows, one or many splits (also more splits than
    a short sequence has pages)."""
    ks = kernel_sets[dtype]
    pos0 = [0, 63, 64, 700, 257]
    B = len(pos0)
    qs, kk, vv = attention_case(H, G, hd, [1] * B, pos0, 44)
    rnd = (lambda t: t) if dtype == torch.float32 else (lambda t: t.bfloat16().float())
    qs, kk, vv = [rnd(t) for t in qs], [rnd(t) for t in kk], [rnd(t) for t in vv]
    kp, vp, bt = paged(kk, vv, [p + 1 for p in pos0], dtype=dtype)
    q = dev(torch.cat([t.reshape(1, -1) for t in qs]), dtype)
    assert ks.attn_decode_split_takes(hd, q.stride(0))
    out = torch.full((B, H * hd), float("nan"), dtype=dtype, device="cuda")
    part = torch.full((B * H * n_split * (hd + 2),), float("nan"), dtype=torch.float32, device="cuda") if n_split > 1 else None
    ks.attn_decode_split(q, out, dev(pos0, torch.int32), bt, kp, vp, part, B, H, G, hd, window, 1.0 / math.sqrt(hd), n_split)
    want = torch.cat([plain.attention(f64(qs[b]), f64(kk[b]), f64(vv[b]), torch.tensor([pos0[b]]),
                                      torch.arange(pos0[b] + 1), window).reshape(1, -1) for b in range(B)])
    assert rel_err(out.cpu().float(), want) < TOL[dtype]


@pytest.mark.parametrize("H, G, hd, vd, n_split", [(9, 1, 32, 64, 1), (14, 2, 24, 40, 3), (64, 1, 32, 64, 2), (6, 2, 64, 256, 2), (10, 2, 320, 64, 1)])
def test_attn_decode_split_of_groups_of_any_size(kernel_sets, H, G, hd, vd, n_split):
    """Groups that fill no block's heads, unequal widths: the attention of every head; and many heads on one key/value head, a block for
    every few of them, take no longer than a block a row and head (one block for all of them took ten times that)."""
    ks, pos0, g = kernel_sets[torch.float32], [0, 63, 130], torch.Generator().manual_seed(H)
    held = [p + 1 for p in pos0]
    kk, vv = [torch.randn(n, G, hd, generator=g) for n in held], [torch.randn(n, G, vd, generator=g) for n in held]
    kp, _, bt = paged(kk, kk, held)
    vp, _, _ = paged(vv, vv, held)
    q = torch.randn(3, H, hd, generator=g)
    out, part = torch.full((3, H * vd), float("nan"), device="cuda"), torch.full((3 * H * n_split * (vd + 2),), float("nan"), device="cuda")
    qd, pd = dev(q.view(3, -1)), dev(pos0, torch.int32)
    split = lambda: ks.attn_decode_split(qd, out, pd, bt, kp, vp, part, 3, H, G, hd, 0, hd ** -0.5, n_split, v_dim=vd)      # noqa: E731
    split()
    want = []
    for b in range(3):
        k, v = (f64(t).repeat_interleave(H // G, 1) for t in (kk[b], vv[b]))
        sc = (torch.einsum("hd,khd->hk", f64(q[b]), k) * hd ** -0.5).softmax(-1)
        want.append(torch.einsum("hk,khd->hd", sc, v).reshape(-1))
    assert rel_err(out.cpu(), torch.stack(want)) < TOL[torch.float32]
    if H // G > 32:
        wide = lambda: ks.seq.attn_wide_value(qd, out, pd, torch.arange(3, dtype=torch.int32, device="cuda"), bt, kp, vp, H, G, hd, vd, 0, hd ** -0.5)      # noqa: E731

        def us(run):
            run()
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                for _ in range(20):
                    run()
            start.record()
            graph.replay()
            end.record()
            torch.cuda.synchronize()
            return start.elapsed_time(end)

        assert us(split) < 3 * us(wide)


FAR_CASES = [(3, None, True), (517, None, True), (899 - 199, 200, True), (899 - 200, 200, False),
             (640, 260, True), (639, 260, False)]     # the last two: the window's edge (key 640) on a page and tile boundary


def far_key_case(H, G, hd, n, far, dtype, n_new=1):
    """`n` keys; the queries at the last `n_new` positions all point at key `far`, whose score towers
    over the others: the output must be that key's value if and only if the key is seen."""
    k = rand(n, G, hd, seed=60, scale=0.1)
    v = rand(n, G, hd, seed=61)
    base = rand(G, hd, seed=62, scale=0.1)                               # one query direction per key/value head
    nrep = H // G
    q = base.repeat_interleave(nrep, dim=0)[None].repeat(n_new, 1, 1).contiguous()    # every head of a group, every row
    k[far] = base * (2260.0 / math.sqrt(hd))                            # score about 22 above the others
    rnd = (lambda t: t) if dtype == torch.float32 else (lambda t: t.bfloat16().float())
    return rnd(q), rnd(k), rnd(v)


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_finds_one_far_key_and_respects_the_windows_edge(kernel_sets, dtype):
    """Random keys would hide a key read from the wrong place: one key among 900 gets a score far
    above the rest, so the output must be that key's value; with a window, the key at distance
    window-1 is seen and the key at distance window is not. Through the generic kernels of both
    element types: the one-query form, the register-tiled form (several new rows on a non-empty
    cache) and the split-key decode form."""
    ks = kernel_sets[dtype]
    H = G = 2
    hd, n = 32, 900
    scale = 1.0 / math.sqrt(hd)
    for far, window, seen in FAR_CASES:
        q, k, v = far_key_case(H, G, hd, n, far, dtype)
        kp, vp, bt = paged([k], [v], [n], dtype=dtype, seed=far)
        out = torch.empty(1, H * hd, dtype=dtype, device="cuda")
        qd = dev(q.reshape(1, -1), dtype)
        ks.attn_paged(qd, out, dev([0, 1], torch.int32), dev([n - 1], torch.int32), bt, kp, vp, 1, 1, H, G, hd, window, scale)
        want = plain.attention(f64(q), f64(k), f64(v), torch.tensor([n - 1]), torch.arange(n), window).reshape(1, -1)
        assert rel_err(out.cpu().float(), want) < TOL[dtype]
        hit = rel_err(out.cpu().float(), f64(v[far]).reshape(1, -1)) < 1e-2
        assert hit == seen
        for n_split in (1, 5):
            part = torch.empty(H * n_split * (hd + 2), dtype=torch.float32, device="cuda")
            out.fill_(float("nan"))
            ks.attn_decode_split(qd, out, dev([n - 1], torch.int32), bt, kp, vp, part, 1, H, G, hd, window, scale, n_split)
            assert rel_err(out.cpu().float(), want) < TOL[dtype]
            assert (rel_err(out.cpu().float(), f64(v[far]).reshape(1, -1)) < 1e-2) == seen
        if dtype == torch.bfloat16:
            for n_split in (1, 5):
                scratch = torch.empty(H * n_split * (hd + 2), dtype=torch.float32, device="cuda")
                ks.decode.attn_decode(qd, out, dev([n - 1], torch.int32), bt, kp, vp, scratch, 1, H, G, hd, window, scale, n_split)
                assert rel_err(out.cpu().float(), want) < TOL[dtype]
                assert (rel_err(out.cpu().float(), f64(v[far]).reshape(1, -1)) < 1e-2) == seen
        # the register-tiled form: the last 7 rows are new, the far key lies in an earlier page of the cache
        n_new = 7
        q7, k7, v7 = far_key_case(H, G, hd, n, far, dtype, n_new)
        out7 = torch.empty(n_new, H * hd, dtype=dtype, device="cuda")
        ks.attn_paged(dev(q7.reshape(n_new, -1), dtype), out7, dev([0, n_new], torch.int32), dev([n - n_new], torch.int32), bt,
                      kp, vp, 1, n_new, H, G, hd, window, scale)
        want7 = plain.attention(f64(q7), f64(k7), f64(v7), torch.arange(n - n_new, n), torch.arange(n), window).reshape(n_new, -1)
        assert rel_err(out7.cpu().float(), want7) < TOL[dtype]
        assert (rel_err(out7[-1:].cpu().float(), f64(v[far]).reshape(1, -1)) < 1e-2) == seen


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("H, G", [(4, 2), (24, 2), (3, 3)])
def test_fast_bfloat16_attention_finds_one_far_key_and_respects_the_windows_edge(kernel_sets, hd, H, G):
    """The same through the kernels that generation uses at real head widths: the tcgen05 prompt
    attention with new rows on a non-empty cache (the far key in an earlier page, the window's edge
    inside a 64-key tile and on a tile boundary), the decode attention on mma.sync with grouped
    queries (4 and 24 heads on 2 key/value heads: its lower rows only, and its upper rows too) and
    its one-head form, with one and five splits, and the decode form that rotates and writes the
    cache itself (identity rotation: position table of angle 0)."""
    ks = kernel_sets[torch.bfloat16]
    n = 900
    scale = 1.0 / math.sqrt(hd)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ident = torch.zeros(n, hd // 2, 2, dtype=torch.float32, device="cuda")
    ident[..., 0] = 1.0                                                  # cos 1, sin 0 at every position
    for far, window, seen in FAR_CASES:
        q, k, v = far_key_case(H, G, hd, n, far, torch.bfloat16)
        kp, vp, bt = paged([k], [v], [n], dtype=torch.bfloat16, seed=far)
        qd = dev(q.reshape(1, -1), torch.bfloat16)
        want = plain.attention(f64(q), f64(k), f64(v), torch.tensor([n - 1]), torch.arange(n), window).reshape(1, -1)
        vfar = torch.cat([f64(v[far, h // (H // G)]) for h in range(H)]).reshape(1, -1)
        tickets = torch.zeros(G, dtype=torch.int32, device="cuda")
        for n_split in (1, 5):
            scratch = torch.empty(H * n_split * (hd + 2), dtype=torch.float32, device="cuda")
            out = torch.full((1, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
            ks.decode.attn_decode(qd, out, dev([n - 1], torch.int32), bt, kp, vp, scratch, 1, H, G, hd, window, scale, n_split,
                                  tickets=tickets)
            assert rel_err(out.cpu().float(), want) < 1.2e-2
            assert (rel_err(out.cpu().float(), vfar) < 1e-2) == seen
            # rotation and cache write fused: raw row [q | k | v] of the last position, the cache holds the rest
            raw = torch.cat([q.reshape(1, -1), k[n - 1].reshape(1, -1), v[n - 1].reshape(1, -1)], dim=1)
            kp2, vp2 = kp.clone(), vp.clone()
            pg = int(bt[0, (n - 1) // PAGE])
            kp2[pg, :, (n - 1) % PAGE] = float("nan")
            vp2[pg, :, (n - 1) % PAGE] = float("nan")
            out.fill_(float("nan"))
            ks.decode.attn_decode_rope(dev(raw, torch.bfloat16), out, dev([n - 1], torch.int32), bt, kp2, vp2, scratch, tickets,
                                       ident, hd, False, True, 1, H, G, hd, window, scale, n_split)
            assert rel_err(out.cpu().float(), want) < 1.2e-2
            assert (rel_err(out.cpu().float(), vfar) < 1e-2) == seen
            assert torch.equal(kp2[pg, :, (n - 1) % PAGE], kp[pg, :, (n - 1) % PAGE])
        # prompt attention: 70 new rows on 830 cached keys; the last row's far key lies pages back
        n_new = 70
        q7, k7, v7 = far_key_case(H, G, hd, n, far, torch.bfloat16, n_new)
        out7 = torch.full((n_new, H * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
        ks.prefill_attention_tc.attn(dev(q7.reshape(n_new, -1), torch.bfloat16), out7, dev([0, n_new], torch.int32),
                                     dev([n - n_new], torch.int32), bt, kp, vp, 1, n_new, H, G, hd, window, scale, err)
        want7 = plain.attention(f64(q7), f64(k7), f64(v7), torch.arange(n - n_new, n), torch.arange(n), window).reshape(n_new, -1)
        assert int(err) == 0
        assert rel_err(out7.cpu().float(), want7) < 1.2e-2
        assert (rel_err(out7[-1:].cpu().float(), vfar) < 1e-2) == seen


# --------------------------------------------------------------------------- sampling
def params_for(options, seeds, draws):
    from scriptling_llm_lib_b200.sampling.sampler import pack_params
    return dev(pack_params(options, seeds, draws))


@pytest.mark.parametrize("V", [5, 384, 1003, 49152])
def test_sampling_kernel_follows_the_plain_samplers(V):
    from scriptling_llm_lib_b200.csrc.bindings import SamplingKernels
    from scriptling_llm_lib_b200.sampling.sampler import SamplingOptions
    sk = SamplingKernels()
    n = 12
    logits = rand(n, V, seed=70, scale=2.5)
    logits[0, 3] = logits[0].max() + 1.0
    if V > 4:
        logits[0, 1] = logits[0, 3]                                     # equal maxima: the first wins
        logits[1, :] = 0.25                                             # all equal but one: ties everywhere
        logits[1, 0] = 0.5
    lg = dev(logits)
    seeds = [1000 + 7 * i for i in range(n)]
    draws = [i % 5 for i in range(n)]
    for opts in [SamplingOptions("greedy"), SamplingOptions("temperature", 0.8), SamplingOptions("temperature", 2.5),
                 SamplingOptions("top_k", 0.9, top_k=7), SamplingOptions("top_k", 1.0, top_k=1),
                 SamplingOptions("top_k", 1.3, top_k=10 ** 6), SamplingOptions("top_p", 1.0, top_p=0.5),
                 SamplingOptions("top_p", 0.7, top_p=0.9), SamplingOptions("top_p", 1.0, top_p=1.0),
                 SamplingOptions("temperature", 0.0)]:
        out = torch.empty(n, dtype=torch.int32, device="cuda")
        sk.sample_rows(lg, params_for(opts, seeds, draws), out)
        got = out.cpu().tolist()
        for i in range(n):
            u = plain.uniform_for(seeds[i], draws[i])
            strategy = "greedy" if opts.is_greedy else opts.strategy
            want = plain.sample(logits[i].numpy(), strategy, opts.temperature or 1.0, opts.top_k, opts.top_p, u)
            assert got[i] == want, f"{opts} row {i}: kernel {got[i]}, plain {want}"
    # a strided view of a wider buffer (the padded logits of a replayed step)
    wide = torch.zeros(n, V + 13, device="cuda")
    wide[:, :V] = lg
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    sk.sample_rows(wide[:, :V], params_for(SamplingOptions("greedy"), seeds, draws), out)
    assert out.cpu().tolist() == [plain.argmax_first(logits[i].numpy()) for i in range(n)]


def test_temperature_sampling_has_the_right_distribution():
    from scriptling_llm_lib_b200.csrc.bindings import SamplingKernels
    from scriptling_llm_lib_b200.sampling.sampler import SamplingOptions
    sk = SamplingKernels()
    logits = torch.tensor([[0.0, 1.0, 2.0, -1.0, 0.5]])
    n = 4000
    lg = dev(logits.repeat(n, 1))
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    sk.sample_rows(lg, params_for(SamplingOptions("temperature", 0.7), [5] * n, list(range(n))), out)
    freq = np.bincount(out.cpu().numpy(), minlength=5) / n
    assert np.abs(freq - plain.softmax_t(logits[0].numpy(), 0.7)).max() < 0.03


def test_repeat_penalty_kernel():
    from scriptling_llm_lib_b200.csrc.bindings import SamplingKernels
    sk = SamplingKernels()
    logits = rand(3, 50, seed=80)
    lg = dev(logits.clone())
    recent = [[4, 9, 4, 49, 60, -1, 9], list(range(30)), [7]]
    last_n = 6
    win = np.full((3, last_n), -1, dtype=np.int32)
    counts = np.zeros(3, dtype=np.int32)
    for i, r in enumerate(recent):
        tail = r[-last_n:]
        win[i, :len(tail)], counts[i] = tail, len(tail)
    pen = dev([1.3, 2.0, 0.0])
    sk.repeat_penalty(lg, dev(win), dev(counts), pen, last_n)
    for i, p in enumerate([1.3, 2.0]):
        want = plain.apply_repeat_penalty(logits[i].numpy(), recent[i], p, last_n)
        assert rel_err(lg[i].cpu(), want) < 1e-6
    assert torch.equal(lg[2].cpu(), logits[2])                           # penalty 0: off

@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("H, G, hd, vd, window, keep, softcap", [(4, 2, 64, 128, 0, 0, None), (3, 3, 80, 80, 100, 0, None), (2, 1, 16, 40, 90, 30, 5.0),
                                                                 (2, 2, 192, 128, 0, 0, None)])
def test_a_value_that_is_not_finite_is_seen_by_the_queries_that_see_it(kernel_sets, H, G, hd, vd, window, keep, softcap, bad):
    """Prompt attention with float weights on tcgen05: one value of one key of either sequence is not finite, in the first, a middle and
    the last page; the outputs that are not finite are those of the queries that see it, in its column, and the others are as they are
    with an ordinary value there, to two roundings of the output."""
    from types import SimpleNamespace
    ks, lens, pos0 = kernel_sets[torch.bfloat16], [300, 130], [70, 0]
    T, ends = sum(lens), [n + p for n, p in zip(lens, pos0)]
    pages = [-(-e // 64) for e in ends]
    table = torch.zeros(2, max(pages), dtype=torch.int32)
    table[0, :pages[0]], table[1, :pages[1]] = torch.arange(pages[0]), torch.arange(pages[0], sum(pages))
    kp, v0 = dev(rand(sum(pages), G, 64, hd, seed=1), torch.bfloat16), dev(rand(sum(pages), G, 64, vd, seed=2), torch.bfloat16)
    q = dev(rand(T, H * hd, seed=3), torch.bfloat16)
    i32 = lambda a: dev(a, torch.int32)      # noqa: E731
    start, err, table = i32([0, lens[0], T]), torch.zeros(1, dtype=torch.int32, device="cuda"), table.cuda()

    def run(v):
        out = torch.full((T, H * vd), 7.0, dtype=torch.bfloat16, device="cuda")
        ks.prefill_attention_tc.attn(q, out, start, i32(pos0), table, kp, v, 2, max(lens), H, G, hd, window, hd ** -0.5, err, softcap=softcap,
                                     keep=keep, v_dim=vd, exact_weights=True)
        return out.view(T, H, vd)
    plain_out = run(v0)
    for at in ((3, 5), (200, 64), (369, 129)):
        v = v0.clone()
        for b in range(2):
            v[int(table[b, at[b] // 64]), G - 1, at[b] % 64, 9] = bad
        out = run(v)
        hit = torch.zeros(T, H, vd, dtype=torch.bool, device="cuda")
        for b, row0 in ((0, 0), (1, lens[0])):
            pos = pos0[b] + torch.arange(lens[b], device="cuda")
            sees = (at[b] <= pos) & ((pos - at[b] < window) | (at[b] < keep) if window else True)
            hit[row0:row0 + lens[b], (G - 1) * (H // G):, 9] = sees[:, None]
        assert int(err) == 0 and bool(hit.any()) and torch.equal(~hit, out.isfinite())
        assert float((out - plain_out)[~hit].abs().max()) <= 2.0 ** -7 * float(plain_out.abs().max())


@pytest.mark.parametrize("blocks, M, N, K", [(10, 1, 512, 256), (5, 8, 20, 24), (3, 17, 256, 72), (2, 32, 512, 256),
                                             (5, 33, 512, 256), (3, 128, 256, 64), (10, 129, 512, 256), (2, 700, 256, 128)])
def test_bfloat16_block_diagonal_products(kernel_sets, blocks, M, N, K):
    """One launch for every block, on a column slice of a wider buffer, from one row to several row tiles: each sum within what K
    additions of exact products can lose, and with few rows the bits of a launch a block."""
    ks, bf = kernel_sets[torch.bfloat16], torch.bfloat16
    wide, w = dev(rand(M, blocks * K + 8, seed=3), bf), dev(rand(blocks, N, K, seed=4), bf)
    a = wide[:, 8:]
    out = torch.full((blocks, M, N), float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    few = ks.decode.takes_blocks(a, w)
    assert few == (M <= 32) and not ks.decode.takes_blocks(wide[:, 1:1 + blocks * K], w)
    if few:
        ks.decode.gemm_small_m_blocks(a, w, out)
        each = torch.empty_like(out)
        for b in range(blocks):
            ks.decode.gemm_small_m(a[:, b * K:(b + 1) * K], w[b], each[b])
        assert torch.equal(out, each)
    else:
        assert ks.tensor_core.takes_blocks(a, w) and not ks.tensor_core.takes_blocks(wide[:, 1:1 + blocks * K], w)
        assert not ks.tensor_core.takes_blocks(a, w[:, :N - 16].contiguous())
        ks.tensor_core.gemm_blocks(a, w, out, err)
    x = f64(a).view(M, blocks, K)
    want = torch.einsum("mbk,bnk->bmn", x, f64(w))
    room = torch.einsum("mbk,bnk->bmn", x.abs(), f64(w).abs()) * (K + 4) * 2.0 ** -23      # an addition cuts at most its last bit
    assert ((f64(out) - want).abs() <= room).all() and err.item() == 0
