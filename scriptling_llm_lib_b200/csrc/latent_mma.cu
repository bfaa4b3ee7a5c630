// Decode attention over a cached latent on mma.sync (bfloat16 engines): the queries that ask the latent, scores and sums over the
// cached rows, and the head's values. One query a sequence and sixteen heads that read the same cached rows are the sixteen rows of
// an mma tile, which tcgen05's 128 would leave seven eighths empty. What is float stays float: a float operand enters a product as
// the sum of three bfloat16 numbers (8 + 8 + 8 bits of mantissa), the other operand (weights, cached rows) is bfloat16 as it is
// stored, sums are float. The tensor cores cut what does not fit a sum's 24 bits off where FMA rounds, so a sum stays on them for a few
// steps only (a page of keys, three steps of a score), smallest parts first, and is added to what came before as floats: against 64
// bits the sums over 4,096 cached latents of 512 dims are 2.7e-7 off (3.7e-7 on the FMA units; 2.0e-6 while one sum ran through all
// keys), the absorbed queries 1.1e-7 (1.7e-7). The float32 set and other widths have the kernels of mix_kernels.cuh.
#include "common.cuh"

namespace lat {

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16* p) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const bf16* p) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
// 16 bytes into shared memory without a register, or zeros
__device__ __forceinline__ void cp16(bf16* dst, const bf16* src, bool there) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// ------------------------------------------------------------------ the queries
// qa[t][h] = scale * [Wuk_h^T q_unrot | q_rot]. A block has 16 rows, one head and 64 of the latent's columns: the matrix's part comes
// into shared memory in one go, a warp takes 16 columns. Both operands are bfloat16; the scale multiplies the float sums.
#define LAT_AC 64
__global__ void __launch_bounds__(128) latent_absorb_mma_kernel(const bf16* __restrict__ q, int ldq, const bf16* __restrict__ wuk,
                                                                float* __restrict__ qa, int T, int H, int D, int P, int R, float scale) {
  extern __shared__ __align__(16) bf16 smb[];      // [D up to a multiple of 16][72]
  constexpr int LD = LAT_AC + 8;
  const int h = blockIdx.y, t0 = blockIdx.x * 16, c0 = blockIdx.z * LAT_AC, Dp = (D + 15) & ~15;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bf16* w = wuk + (size_t)h * D * R + c0;
  for (int i = threadIdx.x; i < Dp * (LAT_AC / 8); i += 128) {
    const int d = i / (LAT_AC / 8), c = (i % (LAT_AC / 8)) * 8;
    const bool there = d < D && c0 + c < R;
    cp16(smb + d * LD + c, there ? w + (size_t)d * R + c : wuk, there);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  const int ra = t0 + g, rb = ra + 8, W = R + P;
  const bf16* qr_a = q + (size_t)ra * ldq + (size_t)h * (D + P);
  const bf16* qr_b = qr_a + (size_t)8 * ldq;
  if (blockIdx.z == 0)
    for (int i = threadIdx.x; i < 16 * P; i += 128) {
      const int r = t0 + i / P, j = i % P;
      if (r < T) qa[((size_t)r * H + h) * W + R + j] = to_f32(q[(size_t)r * ldq + (size_t)h * (D + P) + D + j]) * scale;
    }
  float acc[2][4];
#pragma unroll
  for (int e = 0; e < 4; e++) acc[0][e] = acc[1][e] = 0.f;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const bf16* at = smb + ((lane & 7) + ((lane >> 3) & 1) * 8) * LD + warp * 16 + (lane >> 4) * 8;
#pragma unroll 4
  for (int k = 0; k < Dp; k += 16) {
    const int c = k + 2 * t;
    uint32_t a[4], b[4];
    a[0] = ra < T && c < D ? *(const uint32_t*)(qr_a + c) : 0u;
    a[1] = rb < T && c < D ? *(const uint32_t*)(qr_b + c) : 0u;
    a[2] = ra < T && c + 8 < D ? *(const uint32_t*)(qr_a + c + 8) : 0u;
    a[3] = rb < T && c + 8 < D ? *(const uint32_t*)(qr_b + c + 8) : 0u;
    ldsm4t(b, at + k * LD);
    mma(acc[0], a, b[0], b[1]);
    mma(acc[1], a, b[2], b[3]);
  }
#pragma unroll
  for (int n = 0; n < 2; n++) {
    const int c = c0 + warp * 16 + n * 8 + 2 * t;
    if (c >= R) continue;
    if (ra < T) *(float2*)(qa + ((size_t)ra * H + h) * W + c) = make_float2(acc[n][0] * scale, acc[n][1] * scale);
    if (rb < T) *(float2*)(qa + ((size_t)rb * H + h) * W + c) = make_float2(acc[n][2] * scale, acc[n][3] * scale);
  }
}

// ------------------------------------------------------------------ scores and sums
// A block has one row, sixteen heads and one split of the row's keys, which come a page (64 rows) at a time, the next page on its
// way while this one is worked on. Scores: warp (kg, half) takes every fourth 16 dims of the 576 for 32 keys, its part of the
// queries, split once, in registers; the four groups' sums meet in shared memory. Softmax: two rows a warp, the weights as three
// planes. Sums over the latent: a warp has an eighth of the columns. Keys first_seen(pos, window) .. pos are seen; rows of a page that
// are not are zeros (what the page holds there may be anything). Each split leaves (max, sum, sums) as latent_attn does.
// Bound by the chain of a page (three barriers, 204 products a warp) with one block an SM. Decode steps of 16 heads on 512 + 64 dims,
// this kernel / with absorb, merge and expand: 8 rows of about 4,000 keys 23.5 / 36 us (106 / 147 on the FMA units), one row 9 / 25
// (21 / 65), 32 rows of about 2,000 keys 52 / 70 (257 / 325).
#define LAT_KEYS SLLM_PAGE
struct AttnArgs {
  const float* qa; const bf16* pages;
  const int* tok_pos; const int* tok_seq; const int* block_table;
  int max_pages;
  float* part;
  int H, R, P, n_split, window;
};
template <int NK, int NT>       // 16-dim steps of a score a warp, 8-column tiles of the sums a warp
__global__ void __launch_bounds__(256) latent_attn_mma_kernel(AttnArgs p) {
  extern __shared__ __align__(16) bf16 smb[];
  __shared__ float corr_s[16];
  constexpr int GROUP = 3;
  const int W = p.R + p.P, LD = W + 8;
  constexpr int SL = LAT_KEYS + 4, PL = LAT_KEYS + 8;
  bf16* tiles = smb;                                    // two of [64][LD], and 512 elements of slack behind them
  bf16* pp = tiles + (size_t)2 * LAT_KEYS * LD + 512;   // 3 x [16][PL]
  float* ss = (float*)(pp + 3 * 16 * PL);               // 4 x [16][SL]
  const int row = blockIdx.x, h0 = blockIdx.y * 16, sp = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int pos = p.tok_pos[row], first = first_seen(pos, p.window);
  const int* pt = p.block_table + (size_t)p.tok_seq[row] * p.max_pages;
  const int page0 = first / LAT_KEYS, n_pages = pos / LAT_KEYS + 1 - page0, per = (n_pages + p.n_split - 1) / p.n_split;
  const int lo = page0 + sp * per, hi = min(page0 + n_pages, lo + per);
  const int chunks = W / 8;

  auto fetch = [&](int page) {
    bf16* dst = tiles + (size_t)((page - lo) & 1) * LAT_KEYS * LD;
    const bf16* src = p.pages + (size_t)pt[page] * LAT_KEYS * W;
    for (int i = tid; i < LAT_KEYS * chunks; i += 256) {
      const int r = i / chunks, c = (i % chunks) * 8, key = page * LAT_KEYS + r;
      const bool there = key <= pos && key >= first;
      cp16(dst + r * LD + c, there ? src + (size_t)r * W + c : p.pages, there);
    }
  };
  if (lo < hi) fetch(lo);
  asm volatile("cp.async.commit_group;" ::: "memory");
  // columns W .. LD of either tile and the slack: zeros, whatever a product reads there
  for (int i = tid; i < 2 * LAT_KEYS; i += 256) *(uint4*)(tiles + (size_t)i * LD + W) = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < 64; i += 256) *(uint4*)(tiles + (size_t)2 * LAT_KEYS * LD + i * 8) = make_uint4(0, 0, 0, 0);

  const int kg = warp & 3, half = warp >> 2;
  uint32_t qf[NK][3][4];
  {
    const int ha = h0 + g, hb = ha + 8;
    const float* qr_a = p.qa + ((size_t)row * p.H + ha) * W;
    const float* qr_b = qr_a + (size_t)8 * W;
#pragma unroll
    for (int s = 0; s < NK; s++) {
      const int c = (kg + 4 * s) * 16 + 2 * t;
      const float2 z = make_float2(0.f, 0.f);
      const float2 f0 = ha < p.H && c < W ? *(const float2*)(qr_a + c) : z, f1 = hb < p.H && c < W ? *(const float2*)(qr_b + c) : z;
      const float2 f2 = ha < p.H && c + 8 < W ? *(const float2*)(qr_a + c + 8) : z, f3 = hb < p.H && c + 8 < W ? *(const float2*)(qr_b + c + 8) : z;
      split_pair(f0.x, f0.y, qf[s][0][0], qf[s][1][0], qf[s][2][0]);
      split_pair(f1.x, f1.y, qf[s][0][1], qf[s][1][1], qf[s][2][1]);
      split_pair(f2.x, f2.y, qf[s][0][2], qf[s][1][2], qf[s][2][2]);
      split_pair(f3.x, f3.y, qf[s][0][3], qf[s][1][3], qf[s][2][3]);
    }
  }
  float o[NT][4];
#pragma unroll
  for (int n = 0; n < NT; n++) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  const int srow = 2 * warp + (lane >> 4), skey = (lane & 15) * 4;      // softmax: sixteen lanes a row, four keys a lane
  float m = -INFINITY, l = 0.f;

  for (int page = lo; page < hi; page++) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                    // the page is there, and the other tile is done with
    if (page + 1 < hi) fetch(page + 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const bf16* tile = tiles + (size_t)((page - lo) & 1) * LAT_KEYS * LD;
    {
      float s[4][4];
#pragma unroll
      for (int n = 0; n < 4; n++) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
      const bf16* kr = tile + (size_t)(half * 32 + (lane & 7) + (lane >> 4) * 8) * LD + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int st = 0; st < NK; st += GROUP) {            // sums of a group of steps, smallest part first, added up as floats
        if ((kg + 4 * st) * 16 >= W) break;
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
          uint32_t b[GROUP][4];
          float f[2][4];
#pragma unroll
          for (int e = 0; e < 4; e++) f[0][e] = f[1][e] = 0.f;
#pragma unroll
          for (int k = 0; k < GROUP; k++)
            if (st + k < NK && (kg + 4 * (st + k)) * 16 < W) ldsm4(b[k], kr + (size_t)n * 8 * LD + (kg + 4 * (st + k)) * 16);
#pragma unroll
          for (int part = 2; part >= 0; part--)
#pragma unroll
            for (int k = 0; k < GROUP; k++)
              if (st + k < NK && (kg + 4 * (st + k)) * 16 < W) {
                mma(f[0], qf[st + k][part], b[k][0], b[k][1]);
                mma(f[1], qf[st + k][part], b[k][2], b[k][3]);
              }
#pragma unroll
          for (int e = 0; e < 4; e++) { s[n][e] += f[0][e]; s[n + 1][e] += f[1][e]; }
        }
      }
      float* d = ss + (kg * 16 + g) * SL + half * 32 + 2 * t;
#pragma unroll
      for (int n = 0; n < 4; n++) {
        *(float2*)(d + n * 8) = make_float2(s[n][0], s[n][1]);
        *(float2*)(d + 8 * SL + n * 8) = make_float2(s[n][2], s[n][3]);
      }
    }
    __syncthreads();
    {
      float v[4];
      const float* r = ss + srow * SL + skey;
      const float4 a = *(const float4*)r, b = *(const float4*)(r + 16 * SL), c = *(const float4*)(r + 32 * SL), d = *(const float4*)(r + 48 * SL);
      v[0] = (a.x + b.x) + (c.x + d.x); v[1] = (a.y + b.y) + (c.y + d.y); v[2] = (a.z + b.z) + (c.z + d.z); v[3] = (a.w + b.w) + (c.w + d.w);
      const int key = page * LAT_KEYS + skey;
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (key + e > pos || key + e < first) v[e] = -INFINITY;
      float mx = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
#pragma unroll
      for (int k = 8; k > 0; k >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, k));
      const float mn = fmaxf(m, mx), cor = mn == -INFINITY ? 1.f : expf(m - mn);
      float sum = 0.f;
#pragma unroll
      for (int e = 0; e < 4; e++) {
        v[e] = v[e] == -INFINITY ? 0.f : expf(v[e] - mn);
        sum += v[e];
      }
#pragma unroll
      for (int k = 8; k > 0; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
      l = l * cor + sum;
      m = mn;
      uint2 q[3];
      split_pair(v[0], v[1], q[0].x, q[1].x, q[2].x);
      split_pair(v[2], v[3], q[0].y, q[1].y, q[2].y);
#pragma unroll
      for (int k = 0; k < 3; k++) *(uint2*)(pp + (k * 16 + srow) * PL + skey) = q[k];
      if ((lane & 15) == 0) corr_s[srow] = cor;
    }
    __syncthreads();
    {
      const float ca = corr_s[g], cb = corr_s[g + 8];
      const bf16* vr = tile + (size_t)((lane & 7) + ((lane >> 3) & 1) * 8) * LD + warp * NT * 8 + (lane >> 4) * 8;
      const bf16* pr = pp + ((lane & 7) + ((lane >> 3) & 1) * 8) * PL + (lane >> 4) * 8;
      uint32_t a[3][LAT_KEYS / 16][4];
#pragma unroll
      for (int part = 0; part < 3; part++)
#pragma unroll
        for (int k = 0; k < LAT_KEYS / 16; k++) ldsm4(a[part][k], pr + part * 16 * PL + k * 16);
#pragma unroll
      for (int n = 0; n < NT; n += 2) {                   // the page's sums, smallest part first; what was there, as floats, behind them
        float f[2][4];
#pragma unroll
        for (int e = 0; e < 4; e++) f[0][e] = f[1][e] = 0.f;
        uint32_t b[LAT_KEYS / 16][4];
#pragma unroll
        for (int k = 0; k < LAT_KEYS / 16; k++) ldsm4t(b[k], vr + (size_t)k * 16 * LD + n * 8);
#pragma unroll
        for (int part = 2; part >= 0; part--)
#pragma unroll
          for (int k = 0; k < LAT_KEYS / 16; k++) {
            mma(f[0], a[part][k], b[k][0], b[k][1]);
            mma(f[1], a[part][k], b[k][2], b[k][3]);
          }
#pragma unroll
        for (int e = 0; e < 2; e++) {
          o[n + e][0] = fmaf(o[n + e][0], ca, f[e][0]); o[n + e][1] = fmaf(o[n + e][1], ca, f[e][1]);
          o[n + e][2] = fmaf(o[n + e][2], cb, f[e][2]); o[n + e][3] = fmaf(o[n + e][3], cb, f[e][3]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  const size_t stride = (size_t)p.n_split * (p.R + 2);
  float* base = p.part + (((size_t)row * p.H + h0) * p.n_split + sp) * (p.R + 2);
  if ((lane & 15) == 0 && h0 + srow < p.H) {
    base[srow * stride] = m;
    base[srow * stride + 1] = l;
  }
  if (lo >= hi) return;                                 // a split without keys leaves its sums unwritten
#pragma unroll
  for (int n = 0; n < NT; n++) {
    const int c = (warp * NT + n) * 8 + 2 * t;
    if (c >= p.R) continue;
    if (h0 + g < p.H) *(float2*)(base + g * stride + 2 + c) = make_float2(o[n][0], o[n][1]);
    if (h0 + g + 8 < p.H) *(float2*)(base + (g + 8) * stride + 2 + c) = make_float2(o[n][2], o[n][3]);
  }
}

// ------------------------------------------------------------------ the values
// olat[t][h] = sum_s w_s acc_s / sum_s w_s l_s, w_s = exp(m_s - max m), a block a (row, head); a `sink` joins the denominator once. All
// of a thread's loads, two columns of every split, are asked for before the first is added. Up to 64 splits.
__global__ void __launch_bounds__(256) latent_merge_wide_kernel(const float* __restrict__ part, float* __restrict__ olat, int R, int n_split,
                                                                const float* __restrict__ sink, int H) {
  __shared__ float w_s[64];
  const size_t item = blockIdx.x;
  const float* p0 = part + item * n_split * (R + 2);
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    const float snk = sink ? sink[item % H] : -INFINITY;
    float ms[2], ls[2], mx = snk;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int s = lane + 32 * i;
      const float2 f = s < n_split ? *(const float2*)(p0 + (size_t)s * (R + 2)) : make_float2(-INFINITY, 0.f);
      ms[i] = f.x;
      ls[i] = f.y;
      mx = fmaxf(mx, f.x);
    }
    mx = warp_max(mx);
    float den = 0.f;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      ms[i] = ms[i] > -INFINITY ? expf(ms[i] - mx) : 0.f;
      den += ms[i] * ls[i];                               // a sum that is no number shows, whatever its weight
    }
    den = warp_sum(den);
    if (sink) den += expf(snk - mx);
#pragma unroll
    for (int i = 0; i < 2; i++) w_s[lane + 32 * i] = ms[i] / den;
  }
  __syncthreads();
  for (int c = threadIdx.x * 2; c < R; c += 512) {
    float2 a = make_float2(0.f, 0.f);
    for (int s0 = 0; s0 < n_split; s0 += 16) {
      float2 f[16];
#pragma unroll
      for (int k = 0; k < 16; k++)                      // a split without keys left its sums unwritten: they are not read
        f[k] = s0 + k < n_split && w_s[s0 + k] != 0.f ? *(const float2*)(p0 + (size_t)(s0 + k) * (R + 2) + 2 + c) : make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 16; k++) {
        if (s0 + k >= n_split) break;
        a.x = fmaf(w_s[s0 + k], f[k].x, a.x);
        a.y = fmaf(w_s[s0 + k], f[k].y, a.y);
      }
    }
    *(float2*)(olat + item * R + c) = a;
  }
}

// out[t][h V + v] = Wuv[h V + v] . olat[t][h], times the sigmoid of a gate logit where there is one (gate_mode 1: one a head, 2: one an
// element). A block has 16 rows, one head and 32 of its values; its four warps take a quarter of the latent's columns each, and the
// sums meet in shared memory. A lane reads 16 bytes of a row of the matrix and the same eight columns of the latents: which of them a
// product's step calls its k is up to us, as long as both operands do the same.
#define LAT_EV 32
__global__ void __launch_bounds__(128) latent_expand_mma_kernel(const float* __restrict__ olat, const bf16* __restrict__ wuv,
                                                                bf16* __restrict__ out, int ldo, int T, int H, int V, int R,
                                                                const bf16* __restrict__ gate, int ldg, int gate_mode) {
  __shared__ float red[3][16][LAT_EV + 2];
  const int h = blockIdx.y, t0 = blockIdx.x * 16, v0 = blockIdx.z * LAT_EV;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ra = t0 + g, rb = ra + 8;
  const float* xa = olat + ((size_t)ra * H + h) * R;
  const float* xb = xa + (size_t)8 * H * R;
  const bf16* w = wuv + ((size_t)h * V + v0 + g) * R;
  float acc[4][4];
#pragma unroll
  for (int n = 0; n < 4; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll 2
  for (int k = warp * 32; k < R; k += 128) {             // 32 columns a step, eight a lane
    const int c = k + t * 8;
    const bool in = c < R;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    uint4 b[4];
#pragma unroll
    for (int n = 0; n < 4; n++) b[n] = in && v0 + n * 8 + g < V ? *(const uint4*)(w + (size_t)n * 8 * R + c) : make_uint4(0, 0, 0, 0);
    const float4 a0 = in && ra < T ? *(const float4*)(xa + c) : z, a1 = in && ra < T ? *(const float4*)(xa + c + 4) : z;
    const float4 b0 = in && rb < T ? *(const float4*)(xb + c) : z, b1 = in && rb < T ? *(const float4*)(xb + c + 4) : z;
    uint32_t f[2][3][4];
    split_pair(a0.x, a0.y, f[0][0][0], f[0][1][0], f[0][2][0]);
    split_pair(b0.x, b0.y, f[0][0][1], f[0][1][1], f[0][2][1]);
    split_pair(a0.z, a0.w, f[0][0][2], f[0][1][2], f[0][2][2]);
    split_pair(b0.z, b0.w, f[0][0][3], f[0][1][3], f[0][2][3]);
    split_pair(a1.x, a1.y, f[1][0][0], f[1][1][0], f[1][2][0]);
    split_pair(b1.x, b1.y, f[1][0][1], f[1][1][1], f[1][2][1]);
    split_pair(a1.z, a1.w, f[1][0][2], f[1][1][2], f[1][2][2]);
    split_pair(b1.z, b1.w, f[1][0][3], f[1][1][3], f[1][2][3]);
    float y[4][4];                                       // the step's sums, smallest part first, added up as floats
#pragma unroll
    for (int n = 0; n < 4; n++) y[n][0] = y[n][1] = y[n][2] = y[n][3] = 0.f;
#pragma unroll
    for (int part = 2; part >= 0; part--)
#pragma unroll
      for (int n = 0; n < 4; n++) {
        mma(y[n], f[0][part], b[n].x, b[n].y);
        mma(y[n], f[1][part], b[n].z, b[n].w);
      }
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[n][e] += y[n][e];
  }
  if (warp > 0) {
#pragma unroll
    for (int n = 0; n < 4; n++) {
      *(float2*)&red[warp - 1][g][n * 8 + 2 * t] = make_float2(acc[n][0], acc[n][1]);
      *(float2*)&red[warp - 1][g + 8][n * 8 + 2 * t] = make_float2(acc[n][2], acc[n][3]);
    }
  }
  __syncthreads();
  if (warp > 0) return;
#pragma unroll
  for (int n = 0; n < 4; n++) {
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const int r = s ? rb : ra, v = v0 + n * 8 + 2 * t;
      if (r >= T || v >= V) continue;
      float2 y = make_float2(acc[n][2 * s], acc[n][2 * s + 1]);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        y.x += red[k][g + 8 * s][n * 8 + 2 * t];
        y.y += red[k][g + 8 * s][n * 8 + 2 * t + 1];
      }
      if (gate_mode == 1) {
        const float z = sigmoid_of(to_f32(gate[(size_t)r * ldg + h]));
        y.x *= z; y.y *= z;
      } else if (gate_mode == 2) {
        y.x *= sigmoid_of(to_f32(gate[(size_t)r * ldg + (size_t)h * V + v]));
        y.y *= sigmoid_of(to_f32(gate[(size_t)r * ldg + (size_t)h * V + v + 1]));
      }
      *(__nv_bfloat162*)(out + (size_t)r * ldo + (size_t)h * V + v) = __floats2bfloat162_rn(y.x, y.y);
    }
  }
}

template <typename K>
static cudaError_t allow_smem(K kernel, size_t smem) {
  return smem <= SLLM_SMEM_UNASKED ? cudaSuccess : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}
static inline bool al(const void* p, size_t bytes) { return ((uintptr_t)p % bytes) == 0; }

template <int NK, int NT>
static int attn_launch(const AttnArgs& p, int T, cudaStream_t stream) {
  const size_t smem = ((size_t)2 * LAT_KEYS * (p.R + p.P + 8) + 512 + 3 * 16 * (LAT_KEYS + 8)) * sizeof(bf16) + (size_t)4 * 16 * (LAT_KEYS + 4) * sizeof(float);
  cudaError_t e = allow_smem(latent_attn_mma_kernel<NK, NT>, smem);
  if (e != cudaSuccess) return (int)e;
  latent_attn_mma_kernel<NK, NT><<<dim3(T, (p.H + 15) / 16, p.n_split), 256, smem, stream>>>(p);
  SLLM_RETURN_LAST();
}

}  // namespace lat

// Whether the kernels below take a layer's widths: a head's D + P dims, values of V, a latent of R with a rotated part of P.
SLLM_EXPORT int sllm_latent_mma_takes(int D, int P, int V, int R) {
  return D >= 8 && D <= 256 && V >= 8 && R >= 8 && R <= 512 && P >= 0 && R + P <= 576 && ((D | P | V | R) & 7) == 0;
}

// q [T, ldq] bfloat16 with head h at columns h (D + P); wuk [H D, R] bfloat16; qa float [T, H, R + P].
SLLM_EXPORT int sllm_latent_absorb_mma(const void* q, int ldq, const void* wuk, float* qa, int T, int H, int D, int P, int R, float scale,
                                       cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!sllm_latent_mma_takes(D, P, 8, R) || H < 1 || H > 65535 || (ldq & 1) || !lat::al(q, 4) || !lat::al(wuk, 16) || !lat::al(qa, 8)) return SLLM_ERR_ARG;
  const size_t smem = (size_t)((D + 15) & ~15) * (LAT_AC + 8) * sizeof(bf16);
  cudaError_t e = lat::allow_smem(lat::latent_absorb_mma_kernel, smem);
  if (e != cudaSuccess) return (int)e;
  lat::latent_absorb_mma_kernel<<<dim3((T + 15) / 16, H, (R + LAT_AC - 1) / LAT_AC), 128, smem, stream>>>((const bf16*)q, ldq, (const bf16*)wuk, qa, T, H, D, P, R, scale);
  SLLM_RETURN_LAST();
}

// qa float [T, H, R + P]; pages [pages][64][R + P] bfloat16; part float [T, H, n_split, R + 2].
SLLM_EXPORT int sllm_latent_attn_mma(const float* qa, const void* pages, const int* tok_pos, const int* tok_seq, const int* block_table,
                                     int max_pages, float* part, int T, int H, int R, int P, int n_split, int window, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!sllm_latent_mma_takes(8, P, 8, R) || H < 1 || n_split < 1 || n_split > 65535 || !lat::al(pages, 16) || !lat::al(qa, 8) || !lat::al(part, 8)) return SLLM_ERR_ARG;
  lat::AttnArgs p{qa, (const bf16*)pages, tok_pos, tok_seq, block_table, max_pages, part, H, R, P, n_split, window};
  const int steps = ((R + P + 15) / 16 + 3) / 4;
  if (R <= 128 && steps <= 3) return lat::attn_launch<3, 2>(p, T, stream);
  if (R <= 256 && steps <= 5) return lat::attn_launch<5, 4>(p, T, stream);
  if (R <= 384 && steps <= 7) return lat::attn_launch<7, 6>(p, T, stream);
  return lat::attn_launch<9, 8>(p, T, stream);
}

// part float [T, H, n_split <= 64, R + 2] -> olat float [T, H, R] (scratch) -> out [T, H V] bfloat16; sink float [H] or null; gate logits
// bfloat16, row stride ldg (gate_mode 0: none, 1: [T, H], 2: [T, H V]).
SLLM_EXPORT int sllm_latent_expand_mma(const float* part, float* olat, const void* wuv, void* out, int ldo, int T, int H, int V, int R,
                                       int n_split, const float* sink, const void* gate, int ldg, int gate_mode, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!sllm_latent_mma_takes(8, 0, V, R) || H < 1 || H > 65535 || n_split < 1 || n_split > 64 || (ldo & 1) || !lat::al(part, 8) || !lat::al(olat, 16) ||
      !lat::al(wuv, 16) || !lat::al(out, 4) || gate_mode < 0 || gate_mode > 2 || (gate_mode && !gate))
    return SLLM_ERR_ARG;
  lat::latent_merge_wide_kernel<<<(unsigned)((size_t)T * H), 256, 0, stream>>>(part, olat, R, n_split, sink, H);
  lat::latent_expand_mma_kernel<<<dim3((T + 15) / 16, H, (V + LAT_EV - 1) / LAT_EV), 128, 0, stream>>>(olat, (const bf16*)wuv, (bf16*)out, ldo, T, H, V, R,
                                                                                                      (const bf16*)gate, ldg, gate_mode);
  SLLM_RETURN_LAST();
}
