// Linear recurrences with a matrix state over many rows, in chunks of 128 rows on tcgen05 (bfloat16 engines; everything inside
// is float and enters a product in three bfloat16 parts, see split_mma.cuh).
//
// Linear attention with a fixed decay g per head: S_t = g S_{t-1} + k_t v_t^T, o_t = S_t^T q_t with q, k, v = silu of the
// projection. Inside a chunk that starts with the state S:
//   o_i = g^(i+1) S^T q_i + sum_{j <= i} g^(i-j) (q_i . k_j) v_j,      S <- g^n S + sum_j g^(n-1-j) k_j v_j^T.
//   chunk_lin_states   what every chunk adds to the state (a product over its rows)
//   chunk_lin_pass     the state in front of every chunk, and the state left at the end
//   chunk_lin_scan     every chunk's outputs from the state in front of it and its own rows: q S, q k^T, and the decayed lower
//                      triangle of the latter times v
// A block has one chunk of one head. Keys up to 128 wide and 128 value columns a block, filled up with zeros. The block's 512
// threads make a tile of three planes (silu, decay, splitting) while the product before it runs; thread 0 issues the products.
// Bound by making the tiles: 200 KB of shared memory is one block an SM, so nothing else runs while a block waits for its
// loads or a product (256 threads a block: 155 + 84 us instead of 79 + 39). 3,001 rows, 16 heads of 128 x 128: 129 us for the
// three kernels (760 in pieces of 32 rows on the FMA units, one piece after the other); the six products of three parts are
// 0.29 of them at the tensor cores' rate. Eight sequences, 9,900 rows: 407 us (1,142).
//
// The gated delta rule: S_t = d_t S_{t-1} + k_t u_t^T with u_t = b_t (v_t - d_t S_{t-1}^T k_t), o_t = S_t^T q_t. With c_i the sum of
// log d over a chunk's rows up to and with i, the rows' corrections of one another are a triangular system: L_ij = b_i e^(c_i - c_j)
// (k_i . k_j) for j < i and T = (I + L)^-1 give U = U0 - W S with U0 = T diag(b) V, W = T diag(b e^c) K, S in front of the chunk.
// With P_ij = e^(c_i - c_j) (q_i . k_j) for j <= i and K' = diag(e^(c_n - c)) K everything a chunk does is linear in S:
//   O = (diag(e^c) Q - P W) S + P U0,      S <- (e^(c_n) I - K'^T W) S + K'^T U0 = M S + N.
//   chunk_delta_parts   the four matrices of every chunk, side by side (they do not know S)
//   chunk_delta_pass    S through the chunks one after the other, 32 of its columns a block
//   chunk_delta_out     every chunk's outputs from the S in front of it
// 2,048 rows of 16 heads of 128 x 128: 100 + 50 + 20 us (640 walked row by row, a dependent chain a column of the state); eight
// sequences, 9,900 rows: 420 + 137 + 103 (1,471). The first kernel has taken 4 us more since it watches for what is not finite. The first kernel is bound by its sixteen warps going through nine tiles and eight
// products one after the other with nothing beside them on the SM; that its code is fetched once a block shows in it too (with
// products and the inversion unrolled, and the paths without 16-byte accesses in the same kernel: 130 us, 597 for the eight).
#include "split_mma.cuh"

namespace chunked {
using namespace sm3;

constexpr int Q = TILE, NT = 512, PIECES = Q * Q / 8 / NT;      // rows of a chunk, threads, 8-column pieces of a tile a thread makes

// z / (1 + exp(-z)); the reciprocal is the hardware's with one Newton step (its error is then a float's last place), which is left out
// where it would meet a product beyond float's range
__device__ __forceinline__ float silu_f(float z) {
  const float d = 1.0f + expf(-z);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float near = fmaf(r, fmaf(-d, r, 1.0f), r);
  return z * (d < 1e36f ? near : r);
}

struct LinArgs {
  const bf16* proj; int ld, q_col, k_col, v_col;      // raw projections, one row a token
  const float* decay;                                 // [H]
  float* state;                                       // [slots][H][D][V]
  const int* seq_start; const int* slots;
  float* chunk_state;                                 // [chunks][hs][D][V]
  float* o;                                           // [T][H V]
  int H, D, V;
  int h0, hs;                                         // the launch's heads: the first, and how many
  int* err;
  int vec;                                            // rows, columns and widths allow 16-byte accesses
};

// The chunks of a sequence lie one behind the other from this one on: the ranges of two sequences never meet, because
// ceil(len / Q) <= floor((start + len) / Q) - floor(start / Q) + 1. There are at most T / Q + sequences of them.
__device__ __forceinline__ size_t first_chunk(int start, int b) { return (size_t)(start / Q + b); }

// The 8-column pieces of a 128 x 128 tile that are this thread's: piece u is row (u * NT + tid) / 16, columns 8 ((u * NT + tid) % 16).
__device__ __forceinline__ void fetch(uint4 (&raw)[PIECES], const bf16* src, int ld, int n, int cols, int vec) {
#pragma unroll
  for (int u = 0; u < PIECES; u++) {
    const int i = u * NT + threadIdx.x, r = i >> 4, c = (i & 15) * 8;
    raw[u] = make_uint4(0, 0, 0, 0);
    if (r >= n || c >= cols) continue;
    if (vec) raw[u] = *(const uint4*)(src + (size_t)r * ld + c);
    else {
      bf16* e = (bf16*)&raw[u];
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (c + k < cols) e[k] = src[(size_t)r * ld + c + k];
    }
  }
}
// What is not finite in a row's value (the delta rule: key, step or decay as well) may reach that row and those behind it, but a
// product over a chunk's rows multiplies it by the zeros in front of it too. So it is put into the tile as 0, and the rows that it
// belongs to are made NaN where they are stored: from `row` on, in column c from `col[c]` on (Q: none).
struct Watch { int row, any, col[Q]; };
__device__ __forceinline__ bool finite(float x) { return x * 0.f == 0.f; }
__device__ __forceinline__ bool finite8(const float (&f)[8]) {
  float t = 0.f;
#pragma unroll
  for (int k = 0; k < 8; k++) t = fmaf(f[k], 0.f, t);
  return t == 0.f;
}
__device__ __forceinline__ void open_watch(Watch& w) {
  if (threadIdx.x < Q) w.col[threadIdx.x] = Q;
  if (threadIdx.x == 0) { w.row = Q; w.any = 0; }
}
__device__ __forceinline__ void watch_columns(Watch& w, float (&f)[8], int r, int c) {
  if (finite8(f)) return;
  w.any = 1;
#pragma unroll
  for (int k = 0; k < 8; k++)
    if (!finite(f[k])) { atomicMin(&w.col[c + k], r); f[k] = 0.f; }
}
// row i of what is stored, columns c0 .. c0 + 31
__device__ __forceinline__ void spoil(const Watch& w, uint32_t (&v)[32], int i, int c0) {
  if (w.row == Q && !w.any) return;
#pragma unroll
  for (int k = 0; k < 32; k++)
    if (i >= min(w.row, w.col[c0 + k])) v[k] = 0x7fc00000u;
}

// silu of what was fetched, row r times scale[r] (null: 1), into the tile's planes
__device__ __forceinline__ void put_silu(uint8_t* tile, const uint4 (&raw)[PIECES], const float* scale, Watch* watch = nullptr) {
#pragma unroll
  for (int u = 0; u < PIECES; u++) {
    const int i = u * NT + threadIdx.x, r = i >> 4, c = (i & 15) * 8;
    const float w = scale ? scale[r] : 1.f;
    const __nv_bfloat162* h = (const __nv_bfloat162*)&raw[u];
    float f[8];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      f[2 * k] = silu_f(__low2float(h[k])) * w;
      f[2 * k + 1] = silu_f(__high2float(h[k])) * w;
    }
    if (watch) watch_columns(*watch, f, r, c);
    put8(tile, r, c, f);
  }
}
// a float matrix [rows][ld] into the tile's planes
__device__ __forceinline__ void put_floats(uint8_t* tile, const float* src, int ld, int rows, int cols, int vec) {
  float f[PIECES][8];
#pragma unroll
  for (int u = 0; u < PIECES; u++) {
    const int i = u * NT + threadIdx.x, r = i >> 4, c = (i & 15) * 8;
#pragma unroll
    for (int k = 0; k < 8; k++) f[u][k] = 0.f;
    if (r >= rows || c >= cols) continue;
    const float* p = src + (size_t)r * ld + c;
    if (vec) {
      const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
      f[u][0] = a.x; f[u][1] = a.y; f[u][2] = a.z; f[u][3] = a.w; f[u][4] = b.x; f[u][5] = b.y; f[u][6] = b.z; f[u][7] = b.w;
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (c + k < cols) f[u][k] = p[k];
    }
  }
#pragma unroll
  for (int u = 0; u < PIECES; u++) {
    const int i = u * NT + threadIdx.x;
    put8(tile, i >> 4, (i & 15) * 8, f[u]);
  }
}
// 32 floats of this thread's lane (row) to a row of a float matrix, columns [c0, c0 + 32) as far as there are
__device__ __forceinline__ void store_row(float* dst, const uint32_t (&v)[32], int c0, int cols, int vec) {
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    if (vec) {
      if (c0 + k < cols)
        *(float4*)(dst + c0 + k) = make_float4(__uint_as_float(v[k]), __uint_as_float(v[k + 1]), __uint_as_float(v[k + 2]), __uint_as_float(v[k + 3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (c0 + k + e < cols) dst[c0 + k + e] = __uint_as_float(v[k + e]);
    }
  }
}

// g^n by squaring, in double
__device__ __forceinline__ float power(float g, int n) {
  double r = 1.0, q = (double)g;
  for (; n > 0; n >>= 1) {
    if (n & 1) r *= q;
    q *= q;
  }
  return (float)r;
}
// powers g^0 .. g^Q of the head's decay
__device__ __forceinline__ void fill_powers(float* pw, float g) {
  if (threadIdx.x <= Q) pw[threadIdx.x] = power(g, threadIdx.x);
}

__device__ __forceinline__ uint8_t* aligned_smem(uint8_t* raw) { return (uint8_t*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023); }

constexpr uint32_t LIN_SMEM = 2 * TILE_BYTES + 2 * (Q + 4) * 4 + 16 + 1024;

__global__ void __launch_bounds__(NT, 1) chunk_lin_states_kernel(LinArgs p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int b = blockIdx.z, start = p.seq_start[b], len = p.seq_start[b + 1] - start, r0 = blockIdx.x * Q;
  if (r0 >= len) return;
  uint8_t* ka = aligned_smem(smem_raw);
  uint8_t* va = ka + TILE_BYTES;
  float* pw = (float*)(va + TILE_BYTES);
  float* scale = pw + Q + 4;
  const int n = min(Q, len - r0), vblocks = (p.V + Q - 1) / Q, hl = blockIdx.y / vblocks, h = p.h0 + hl, v0 = (blockIdx.y % vblocks) * Q;
  const int vn = min(Q, p.V - v0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bf16* row = p.proj + (size_t)(start + r0) * p.ld;
  uint4 kr[PIECES], vr[PIECES];
  fetch(kr, row + p.k_col + (size_t)h * p.D, p.ld, n, p.D, p.vec);
  fetch(vr, row + p.v_col + (size_t)h * p.V + v0, p.ld, n, vn, p.vec);
  fill_powers(pw, p.decay[h]);
  Unit u;
  u.open((uint8_t*)(scale + Q + 4));
  pdl_launch_dependents();               // (behind the allocation: a dependent's block must not take the columns first)
  if (tid < Q) scale[tid] = tid < n ? pw[n - 1 - tid] : 0.f;
  put_silu(va, vr, nullptr);
  __syncthreads();
  put_silu(ka, kr, scale);
  u.ready();
  if (tid < 32) {
    product<true, true>(u.tmem, smem_u32(ka), smem_u32(va), (n + 15) / 16);
    u.commit();
  }
  u.done();
  const int d = (warp & 3) * 32 + lane;
  float* dst = p.chunk_state + (((first_chunk(start, b) + blockIdx.x) * p.hs + hl) * p.D + d) * (size_t)p.V + v0;
  const int c0 = (warp >> 2) * 32;                 // a warp reads 32 lanes (rows) of 32 columns
  uint32_t v[32];
  tmem_ld32(u.tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0, v);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  if (d < p.D) store_row(dst, v, c0, vn, p.vec);
  u.close(p.err);
}

// Per element of a head's state, over the chunks in order: what a chunk adds is replaced by the state in front of it. E elements
// a thread (4 where they come in fours).
template <int E>
__global__ void __launch_bounds__(256) chunk_lin_pass_kernel(LinArgs p) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.z, h = p.h0 + blockIdx.y, start = p.seq_start[b], len = p.seq_start[b + 1] - start;
  const int DV = p.D * p.V, e0 = (blockIdx.x * 256 + threadIdx.x) * E;
  if (e0 >= DV || len <= 0) return;
  const int chunks = (len + Q - 1) / Q;
  const size_t stride = (size_t)p.hs * DV;
  float* u = p.chunk_state + (first_chunk(start, b) * p.hs + blockIdx.y) * (size_t)DV + e0;
  float* st = p.state + ((size_t)p.slots[b] * p.H + h) * DV + e0;
  const float g = p.decay[h], whole = power(g, Q), last = power(g, len - (chunks - 1) * Q);
  float s[E];
#pragma unroll
  for (int e = 0; e < E; e++) s[e] = st[e];
  constexpr int AHEAD = 8;
  for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
    float add[AHEAD][E];
#pragma unroll
    for (int k = 0; k < AHEAD; k++)
      if (c0 + k < chunks) {
        if constexpr (E == 4) {
          const float4 q = *(const float4*)(u + (c0 + k) * stride);
          add[k][0] = q.x; add[k][1] = q.y; add[k][2] = q.z; add[k][3] = q.w;
        } else {
#pragma unroll
          for (int e = 0; e < E; e++) add[k][e] = u[(c0 + k) * stride + e];
        }
      }
#pragma unroll
    for (int k = 0; k < AHEAD; k++)
      if (c0 + k < chunks) {
        if constexpr (E == 4) *(float4*)(u + (c0 + k) * stride) = make_float4(s[0], s[1], s[2], s[3]);
        else {
#pragma unroll
          for (int e = 0; e < E; e++) u[(c0 + k) * stride + e] = s[e];
        }
        const float f = c0 + k == chunks - 1 ? last : whole;
#pragma unroll
        for (int e = 0; e < E; e++) s[e] = fmaf(f, s[e], add[k][e]);
      }
  }
#pragma unroll
  for (int e = 0; e < E; e++) st[e] = s[e];
}

// Tensor memory: q S in columns 0-127; q k^T in 128-255, whose place (and 64 columns more) its decayed lower triangle takes in
// three planes; that times v in 320-447.
__global__ void __launch_bounds__(NT, 1) chunk_lin_scan_kernel(LinArgs p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int b = blockIdx.z, start = p.seq_start[b], len = p.seq_start[b + 1] - start, r0 = blockIdx.x * Q;
  if (r0 >= len) return;
  uint8_t* qa = aligned_smem(smem_raw);
  uint8_t* xa = qa + TILE_BYTES;                   // the state, then the keys, then the values
  float* pw = (float*)(xa + TILE_BYTES);
  __shared__ Watch watch;
  const int n = min(Q, len - r0), vblocks = (p.V + Q - 1) / Q, hl = blockIdx.y / vblocks, h = p.h0 + hl, v0 = (blockIdx.y % vblocks) * Q;
  const int vn = min(Q, p.V - v0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bf16* row = p.proj + (size_t)(start + r0) * p.ld;
  uint4 raw[PIECES];
  fetch(raw, row + p.q_col + (size_t)h * p.D, p.ld, n, p.D, p.vec);
  fill_powers(pw, p.decay[h]);
  open_watch(watch);
  Unit u;
  u.open((uint8_t*)(pw + 2 * (Q + 4)));
  pdl_launch_dependents();               // (behind the allocation: a dependent's block must not take the columns first)
  put_silu(qa, raw, nullptr);
  put_floats(xa, p.chunk_state + ((first_chunk(start, b) + blockIdx.x) * p.hs + hl) * (size_t)p.D * p.V + v0, p.V, p.D, vn, p.vec);
  u.ready();
  const int dsteps = (p.D + 15) / 16, rsteps = (n + 15) / 16;
  if (tid < 32) {
    product<false, true>(u.tmem, smem_u32(qa), smem_u32(xa), dsteps);
    u.commit();
  }
  fetch(raw, row + p.k_col + (size_t)h * p.D, p.ld, n, p.D, p.vec);
  u.done();
  put_silu(xa, raw, nullptr);
  u.ready();
  if (tid < 32) {
    product<false, false>(u.tmem + 128, smem_u32(qa), smem_u32(xa), dsteps);
    u.commit();
  }
  fetch(raw, row + p.v_col + (size_t)h * p.V + v0, p.ld, n, vn, p.vec);
  u.done();
  const int i = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;       // a warp has 32 rows (lanes) and 32 columns
  const uint32_t t_lane = u.tmem + ((uint32_t)((warp & 3) * 32) << 16);
  {
    uint32_t s[32];
    tmem_ld32(t_lane + 128 + c0, s);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    put_silu(xa, raw, nullptr, &watch);            // the keys have been read
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                               // every warp holds its scores: the planes may go over them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t part[3][16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const int j = c0 + 2 * k;
      const float f0 = j <= i ? __uint_as_float(s[2 * k]) * pw[max(i - j, 0)] : 0.f;
      const float f1 = j + 1 <= i ? __uint_as_float(s[2 * k + 1]) * pw[max(i - j - 1, 0)] : 0.f;
      split_pair(f0, f1, part[0][k], part[1][k], part[2][k]);
    }
#pragma unroll
    for (int q = 0; q < 3; q++) tmem_st16(t_lane + 128 + q * 64 + c0 / 2, part[q]);
  }
  u.ready();
  if (tid < 32) {
    product_ta<true>(u.tmem + 320, u.tmem + 128, smem_u32(xa), rsteps);
    u.commit();
  }
  u.done();
  const float f = pw[i + 1];
  float* dst = p.o + ((size_t)(start + r0 + i) * p.H + h) * p.V + v0;
  uint32_t a[32], c[32];
  tmem_ld32(t_lane + c0, a);
  tmem_ld32(t_lane + 320 + c0, c);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 32; k++) c[k] = __float_as_uint(fmaf(f, __uint_as_float(a[k]), __uint_as_float(c[k])));
  spoil(watch, c, i, c0);
  if (i < n) store_row(dst, c, c0, vn, p.vec);
  u.close(p.err);
}

// ------------------------------------------------------------------ the gated delta rule
struct DeltaArgs {
  const float* qk; int ld_qk;                         // rows [G dk queries | G dk keys]
  const float* v; int ld_v;                           // [T][H dv]
  const float* bd;                                    // [T][2 H + G]: b | d | (not read here)
  float* state;                                       // [slots][H][dk][dv]
  const int* seq_start; const int* slots;
  uint8_t* m;                                         // [chunks][hs]: M as the three planes of a tile
  float *n, *qp, *o0;                                 // [chunks][hs][32][128][4] each (see `quad`); n becomes the state in front of the chunk
  float* o;                                           // [T][H dv]
  int H, G, dk, dv;
  int h0, hs;                                         // the launch's heads: the first, and how many
  int* err;
};
constexpr size_t MAT = (size_t)Q * Q;
constexpr int LT = Q + 4;                             // padded row of a float matrix in shared memory
constexpr uint32_t DELTA_SMEM = 2 * TILE_BYTES + 6 * Q * 4 + 16 + 1024;

// A matrix that only these kernels read lies four columns at a time, all rows of a four side by side: a thread that has a row
// (its lane of tensor memory) writes 16 bytes next to its neighbour's. Columns c (a multiple of 4) to c + 3 of row i:
__device__ __forceinline__ size_t quad(int i, int c) { return ((size_t)(c >> 2) * Q + i) * 4; }
__device__ __forceinline__ float4 four(const uint32_t (&v)[32], int k) {
  return make_float4(__uint_as_float(v[k]), __uint_as_float(v[k + 1]), __uint_as_float(v[k + 2]), __uint_as_float(v[k + 3]));
}
__device__ __forceinline__ void store_quads(float* mat, int i, int c0, const uint32_t (&v)[32]) {
#pragma unroll
  for (int k = 0; k < 32; k += 4) *(float4*)(mat + quad(i, c0 + k)) = four(v, k);
}
// such a matrix into a tile's planes: neighbouring threads have neighbouring rows
__device__ __forceinline__ void fetch_quads(float (&f)[PIECES][8], const float* mat) {
#pragma unroll
  for (int u = 0; u < PIECES; u++) {
    const int r = threadIdx.x & (Q - 1), c = ((threadIdx.x >> 7) + u * (NT >> 7)) * 8;
    const float4 a = *(const float4*)(mat + quad(r, c)), b = *(const float4*)(mat + quad(r, c + 4));
    f[u][0] = a.x; f[u][1] = a.y; f[u][2] = a.z; f[u][3] = a.w; f[u][4] = b.x; f[u][5] = b.y; f[u][6] = b.z; f[u][7] = b.w;
  }
}
__device__ __forceinline__ void put_quads(uint8_t* tile, const float (&f)[PIECES][8]) {
#pragma unroll
  for (int u = 0; u < PIECES; u++) put8(tile, threadIdx.x & (Q - 1), ((threadIdx.x >> 7) + u * (NT >> 7)) * 8, f[u]);
}
// This thread's pieces of a float matrix of whole rows; rows from n and columns from `cols` on are zero. Fetching apart from what
// follows, so that the loads are under way while a product runs.
template <bool VEC>
__device__ __forceinline__ void fetch_rows(float (&f)[PIECES][8], const float* src, size_t ld, int n, int cols) {
#pragma unroll
  for (int u = 0; u < PIECES; u++) {
    const int i = u * NT + threadIdx.x, r = i >> 4, c = (i & 15) * 8;
#pragma unroll
    for (int k = 0; k < 8; k++) f[u][k] = 0.f;
    if (r >= n || c >= cols) continue;
    const float* p = src + (size_t)r * ld + c;
    if constexpr (VEC) {
      const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
      f[u][0] = a.x; f[u][1] = a.y; f[u][2] = a.z; f[u][3] = a.w; f[u][4] = b.x; f[u][5] = b.y; f[u][6] = b.z; f[u][7] = b.w;
    } else {
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (c + k < cols) f[u][k] = p[k];
    }
  }
}
__device__ __forceinline__ void clear_rows(float (&f)[PIECES][8]) {
#pragma unroll
  for (int u = 0; u < PIECES; u++)
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (!finite(f[u][k])) f[u][k] = 0.f;
}

// the pieces, row r times scale[r], into the tile's planes
enum { UNWATCHED, BY_ROW, BY_COLUMN };
template <bool SCALED, int WATCHED = UNWATCHED>
__device__ __forceinline__ void put_rows(uint8_t* tile, float (&f)[PIECES][8], const float* scale, Watch* watch = nullptr) {
#pragma unroll
  for (int u = 0; u < PIECES; u++) {
    const int i = u * NT + threadIdx.x, r = i >> 4;
    if constexpr (WATCHED == BY_COLUMN) watch_columns(*watch, f[u], r, (i & 15) * 8);
    if constexpr (WATCHED == BY_ROW) {
      if (!finite8(f[u])) {
        atomicMin(&watch->row, r);
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (!finite(f[u][k])) f[u][k] = 0.f;
      }
    }
    if constexpr (SCALED) {
      const float w = scale[r];
#pragma unroll
      for (int k = 0; k < 8; k++) f[u][k] *= w;
    }
    put8(tile, r, (i & 15) * 8, f[u]);
  }
}
// this thread's 32 floats of row i from column c0 on into a tile's planes
__device__ __forceinline__ void put_lane(uint8_t* tile, int i, int c0, const uint32_t (&v)[32]) {
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; e++) f[e] = __uint_as_float(v[k + e]);
    put8(tile, i, c0 + k, f);
  }
}
// the same into three planes of 64 columns of tensor memory (an A operand)
__device__ __forceinline__ void put_tmem(uint32_t t_lane, int c0, const uint32_t (&v)[32]) {
  uint32_t part[3][16];
#pragma unroll
  for (int k = 0; k < 16; k++)
    split_pair(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]), part[0][k], part[1][k], part[2][k]);
#pragma unroll
  for (int q = 0; q < 3; q++) tmem_st16(t_lane + q * 64 + c0 / 2, part[q]);
}
// the same into a float matrix in shared memory, and whole rows of that to memory
__device__ __forceinline__ void stage_lane(float* t, int i, int c0, const uint32_t (&v)[32]) {
#pragma unroll
  for (int k = 0; k < 32; k += 4) *(float4*)(t + i * LT + c0 + k) = four(v, k);
}
template <bool VEC>
__device__ __forceinline__ void write_rows(const float* t, float* dst, size_t ld, int n, int cols) {
  const int c = (threadIdx.x & 31) * 4;
#pragma unroll 1
  for (int r = threadIdx.x >> 5; r < n; r += NT / 32) {
    const float4 f = *(const float4*)(t + r * LT + c);
    float* d = dst + (size_t)r * ld + c;
    if constexpr (VEC) {
      if (c < cols) *(float4*)d = f;
    } else {
      if (c < cols) d[0] = f.x;
      if (c + 1 < cols) d[1] = f.y;
      if (c + 2 < cols) d[2] = f.z;
      if (c + 3 < cols) d[3] = f.w;
    }
  }
}
__device__ __forceinline__ void take(uint32_t t_addr, uint32_t (&v)[32]) {
  tmem_ld32(t_addr, v);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// One level of the inversion: pairs of neighbouring S x S blocks on the diagonal that are inverted already, T11 and T22, and L21
// below the first become -T22 L21 T11 there. A warp has 16 x 16 elements of one pair's block, split on their way out of shared
// memory; blocks this small would leave tcgen05's 128 rows empty, and on the FMA units their operands' reads from shared memory
// took 24,000 of a block's 85,000 cycles (16,000 so).
template <int S>
__device__ __forceinline__ void merge_level(float* t) {
  constexpr int SIDE = S / 16, TILES = SIDE * SIDE * (64 / S);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = (lane & 3) * 2;
  const int o = warp / (SIDE * SIDE) * 2 * S, i0 = warp % (SIDE * SIDE) / SIDE * 16, j0 = warp % SIDE * 16;
  const float *t11 = t + o * LT + o, *t22 = t + (o + S) * LT + o + S;
  float* l21 = t + (o + S) * LT + o;
#pragma unroll 1
  for (int side = 0; side < 2; side++) {             // first L21 T11, then T22 times that
    float acc[2][4];
#pragma unroll
    for (int e = 0; e < 4; e++) acc[0][e] = acc[1][e] = 0.f;
    if (warp < TILES) {
      const float *lhs = (side ? t22 : l21) + (i0 + g) * LT, *rhs = (side ? l21 : t11) + j0 + g;
#pragma unroll 1
      for (int k = 0; k < S; k += 16) {
        uint32_t a[3][4], b[2][3][2];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float2 f = *(const float2*)(lhs + (e & 1) * 8 * LT + k + (e >> 1) * 8 + q);
          split_pair(f.x, f.y, a[0][e], a[1][e], a[2][e]);
        }
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const float* r = rhs + (k + e * 8 + q) * LT + n * 8;
            split_pair(r[0], r[LT], b[n][0][e], b[n][1][e], b[n][2][e]);
          }
#pragma unroll
        for (int n = 0; n < 2; n++) {
          mma_bf16(acc[n], a[2], b[n][0]);
          mma_bf16(acc[n], a[0], b[n][2]);
          mma_bf16(acc[n], a[1], b[n][1]);
          mma_bf16(acc[n], a[1], b[n][0]);
          mma_bf16(acc[n], a[0], b[n][1]);
          mma_bf16(acc[n], a[0], b[n][0]);
        }
      }
    }
    __syncthreads();
    if (warp < TILES) {
      const float sign = side ? -1.f : 1.f;
#pragma unroll
      for (int n = 0; n < 2; n++) {
        float* d = l21 + (i0 + g) * LT + j0 + n * 8 + q;
        *(float2*)d = make_float2(sign * acc[n][0], sign * acc[n][1]);
        *(float2*)(d + 8 * LT) = make_float2(sign * acc[n][2], sign * acc[n][3]);
      }
    }
    __syncthreads();
  }
}

// Tensor memory: k k^T in columns 0-127 and q k^T in 128-255, later T in three planes 0-191 and P in 192-383; sums in 384-511 (and,
// once T is done with, in 0-127). VEC: 16-byte accesses are allowed everywhere.
template <bool VEC>
__global__ void __launch_bounds__(NT, 1) chunk_delta_parts_kernel(DeltaArgs p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int b = blockIdx.z, start = p.seq_start[b], len = p.seq_start[b + 1] - start, r0 = blockIdx.x * Q;
  if (r0 >= len) return;
  uint8_t* xa = aligned_smem(smem_raw);            // keys, then K', then M
  uint8_t* ya = xa + TILE_BYTES;                   // queries, L and T as floats, scaled values, U0, scaled keys, W, scaled queries as floats
  float* t = (float*)ya;
  float *hi = (float*)(ya + TILE_BYTES), *lo = hi + Q, *beta = lo + Q, *front = beta + Q, *back = front + Q, *bfront = back + Q;
  __shared__ double part_s[4];
  __shared__ Watch watch;
  const int n = min(Q, len - r0), row = start + r0, h = p.h0 + blockIdx.y, g = h / (p.H / p.G);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* qrow = p.qk + (size_t)row * p.ld_qk + (size_t)g * p.dk;
  const float* krow = qrow + (size_t)p.G * p.dk;
  const float* vrow = p.v + (size_t)row * p.ld_v + (size_t)h * p.dv;
  float f[PIECES][8];
  fetch_rows<VEC>(f, krow, p.ld_qk, n, p.dk);
  open_watch(watch);
  Unit u;
  u.open((uint8_t*)(bfront + Q));
  pdl_launch_dependents();               // (behind the allocation: a dependent's block must not take the columns first)
  // a thread a row: the running sum of log2 d, in double; a decay of 0 is far below what a float can hold from one row to the next
  double c = 0.0;
  float bt = 0.f;
  if (tid < Q) {
    if (tid < n) {
      const float* e = p.bd + (size_t)(row + tid) * (2 * p.H + p.G) + h;
      bt = e[0];
      c = log2((double)e[p.H]);
      if (c < -1000.0) c = -1000.0;
      if (!finite(bt) || !(c <= 1000.0)) {
        atomicMin(&watch.row, tid);
        bt = 0.f;
        c = 0.0;
      }
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double w = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) c += w;
    }
    if (lane == 31) part_s[warp] = c;
  }
  put_rows<false, BY_ROW>(xa, f, nullptr, &watch);
  u.ready();
  const int dsteps = (p.dk + 15) / 16;
  if (tid < 32) {
    product<false, false>(u.tmem, smem_u32(xa), smem_u32(xa), dsteps);
    u.commit();
  }
  fetch_rows<VEC>(f, qrow, p.ld_qk, n, p.dk);
  double last = 0.0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (k < warp && tid < Q) c += part_s[k];
    last += part_s[k];
  }
  if (tid < Q) {
    const float ch = (float)c;
    hi[tid] = ch;
    lo[tid] = (float)(c - (double)ch);
    beta[tid] = bt;
    front[tid] = exp2f(ch);
    back[tid] = exp2f((float)(last - c));
    bfront[tid] = bt * exp2f(ch);
  }
  const float whole = exp2f((float)last);
  put_rows<false>(ya, f, nullptr);
  u.done();
  u.ready();
  if (tid < 32) {
    product<false, false>(u.tmem + 128, smem_u32(ya), smem_u32(xa), dsteps);
    u.commit();
  }
  fetch_rows<VEC>(f, krow, p.ld_qk, n, p.dk);
  u.done();
  if (watch.row < Q) clear_rows(f);
  put_rows<true>(xa, f, back);
  const int i = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;       // a warp has 32 rows (lanes) and 32 columns
  const uint32_t t_lane = u.tmem + ((uint32_t)((warp & 3) * 32) << 16);
  {
    uint32_t s1[32], s2[32];
    tmem_ld32(t_lane + c0, s1);
    take(t_lane + 128 + c0, s2);
    const float hii = hi[i], loi = lo[i], bi = beta[i];
#pragma unroll
    for (int k = 0; k < 32; k++) {
      const int j = c0 + k;
      const float e = j <= i ? exp2f((hii - hi[j]) + (loi - lo[j])) : 0.f;
      s2[k] = __float_as_uint(j <= i ? e * __uint_as_float(s2[k]) : 0.f);
      s1[k] = __float_as_uint(j < i ? bi * (e * __uint_as_float(s1[k])) : 0.f);
    }
    stage_lane(t, i, c0, s1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                               // every warp holds its scores: P may go over them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    put_tmem(t_lane + 192, c0, s2);
  }
  // T = (I + L)^-1 in place: 16 x 16 blocks on the diagonal, a thread a column, then neighbours merged three times
  if (tid < Q) {
    float* d = t + (tid & ~15) * LT + (tid & ~15);
    const int j = tid & 15;
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; r++) {
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 16; k++)
        if (k < r) acc = fmaf(d[r * LT + k], x[k], acc);
      x[r] = r == j ? 1.f : -acc;
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 16; r++) d[r * LT + j] = r < j ? 0.f : x[r];
  }
  __syncthreads();
  merge_level<16>(t);
  merge_level<32>(t);
  fetch_rows<VEC>(f, vrow, p.ld_v, n, p.dv);
  merge_level<64>(t);
  uint32_t w[32];
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const float4 e = *(const float4*)(t + i * LT + c0 + k);
    w[k] = __float_as_uint(e.x); w[k + 1] = __float_as_uint(e.y); w[k + 2] = __float_as_uint(e.z); w[k + 3] = __float_as_uint(e.w);
  }
  put_tmem(t_lane, c0, w);
  __syncthreads();                                 // T has been read from where the scaled values go
  const size_t unit = (first_chunk(start, b) + blockIdx.x) * p.hs + blockIdx.y, mat = unit * MAT;
  put_rows<true, BY_COLUMN>(ya, f, beta, &watch);
  u.ready();
  if (tid < 32) {                                  // U0
    product_ta<true>(u.tmem + 384, u.tmem, smem_u32(ya), 8);
    u.commit();
  }
  u.done();
  take(t_lane + 384 + c0, w);
  put_lane(ya, i, c0, w);
  u.ready();
  if (tid < 32) {                                  // P U0
    product_ta<true>(u.tmem + 384, u.tmem + 192, smem_u32(ya), 8);
    u.commit();
  }
  fetch_rows<VEC>(f, krow, p.ld_qk, n, p.dk);
  u.done();
  take(t_lane + 384 + c0, w);
  u.ready();                                       // the sums have been read
  if (tid < 32) {                                  // K'^T U0
    product<true, true>(u.tmem + 384, smem_u32(xa), smem_u32(ya), 8);
    u.commit();
  }
  spoil(watch, w, i, c0);
  store_quads(p.o0 + mat, i, c0, w);
  u.done();
  if (watch.row < Q) clear_rows(f);
  put_rows<true>(ya, f, bfront);
  take(t_lane + 384 + c0, w);
  u.ready();
  if (tid < 32) {                                  // W
    product_ta<true>(u.tmem + 384, u.tmem, smem_u32(ya), 8);
    u.commit();
  }
  spoil(watch, w, Q - 1, c0);                      // the state behind the chunk has seen all its rows
  store_quads(p.n + mat, i, c0, w);
  u.done();
  take(t_lane + 384 + c0, w);
  put_lane(ya, i, c0, w);
  u.ready();
  if (tid < 32) {                                  // P W and K'^T W
    product_ta<true>(u.tmem + 384, u.tmem + 192, smem_u32(ya), 8);
    product<true, true>(u.tmem, smem_u32(xa), smem_u32(ya), 8);
    u.commit();
  }
  fetch_rows<VEC>(f, qrow, p.ld_qk, n, p.dk);
  u.done();
#pragma unroll
  for (int k = 0; k < PIECES; k++) {               // diag(e^c) Q, from whole rows to a row a thread
    const int e = k * NT + tid, r = e >> 4, cc = (e & 15) * 8;
    const float fr = front[r];
    *(float4*)(t + r * LT + cc) = make_float4(fr * f[k][0], fr * f[k][1], fr * f[k][2], fr * f[k][3]);
    *(float4*)(t + r * LT + cc + 4) = make_float4(fr * f[k][4], fr * f[k][5], fr * f[k][6], fr * f[k][7]);
  }
  take(t_lane + c0, w);
#pragma unroll
  for (int k = 0; k < 32; k++) w[k] = __float_as_uint((i == c0 + k ? whole : 0.f) - __uint_as_float(w[k]));
  put_lane(xa, i, c0, w);
  u.ready();
  if (tid == 0) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(p.m + unit * TILE_BYTES), "r"(smem_u32(xa)), "r"(TILE_BYTES) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  take(t_lane + 384 + c0, w);
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const float4 e = *(const float4*)(t + i * LT + c0 + k);
    w[k] = __float_as_uint(e.x - __uint_as_float(w[k]));
    w[k + 1] = __float_as_uint(e.y - __uint_as_float(w[k + 1]));
    w[k + 2] = __float_as_uint(e.z - __uint_as_float(w[k + 2]));
    w[k + 3] = __float_as_uint(e.w - __uint_as_float(w[k + 3]));
  }
  store_quads(p.qp + mat, i, c0, w);
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  u.close(p.err);
}

// S <- M S + N through a sequence's chunks for 32 columns of a head's state. A thread has a row of 16 columns in registers; their
// three planes, S^T, are the product's second operand (32 rows, two blocks of 64 columns), M's planes come by bulk copies two chunks
// ahead. Bound by the chain of a chunk: split, product (48 steps that read 4 KB of M each), sums back to registers. On the FMA
// units, 16 columns a block, reading M from shared memory took 73 us where this takes 50 (16 chunks).
constexpr int PV = 32;
constexpr uint32_t ST_BLOCK = PV * 128, ST_PLANE = 2 * ST_BLOCK, PASS_SMEM = 2 * TILE_BYTES + 3 * ST_PLANE + 32 + 1024;
__global__ void __launch_bounds__(256, 1) chunk_delta_pass_kernel(DeltaArgs p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ma = aligned_smem(smem_raw);
  uint8_t* sa = ma + 2 * TILE_BYTES;
  uint8_t* head = sa + 3 * ST_PLANE;
  const int b = blockIdx.z, h = p.h0 + blockIdx.y, start = p.seq_start[b], len = p.seq_start[b + 1] - start;
  if (len <= 0) return;
  const int chunks = (len + Q - 1) / Q, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int d = (warp & 3) * 32 + lane, j0 = (warp >> 2) * 16, v0 = blockIdx.x * PV + j0;
  const size_t first = first_chunk(start, b) * p.hs + blockIdx.y;
  float* st = p.state + (((size_t)p.slots[b] * p.H + h) * p.dk + d) * p.dv + v0;
  float* nm = p.n + first * MAT + quad(d, v0);      // columns v0 .. v0 + 15: fours Q * 4 floats apart
  const size_t stride = (size_t)p.hs * MAT;
  const uint32_t full = smem_u32(head + 16);        // two barriers of M's copies
  if (tid == 0) { mbar_init(full, 1); mbar_init(full + 8, 1); }
  Unit u;
  u.open(head);
  pdl_launch_dependents();               // (behind the allocation: a dependent's block must not take the columns first)
  auto fetch_m = [&](int c) {
    const uint32_t bar = full + 8 * (c & 1);
    mbar_expect_tx(bar, TILE_BYTES);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(ma + (c & 1) * TILE_BYTES)), "l"(p.m + (first + (size_t)c * p.hs) * TILE_BYTES), "r"(TILE_BYTES), "r"(bar) : "memory");
  };
  if (tid == 0) {
    fetch_m(0);
    if (chunks > 1) fetch_m(1);
  }
  float own[16];
  float4 add[4];
#pragma unroll
  for (int e = 0; e < 16; e++) own[e] = d < p.dk && v0 + e < p.dv ? st[e] : 0.f;
#pragma unroll
  for (int e = 0; e < 4; e++) add[e] = *(const float4*)(nm + e * Q * 4);
  constexpr uint32_t id = umma_idesc_bf16(128, PV);
  int fetched = min(chunks, 2);                     // copies of M asked for (thread 0's count)
  for (int c = 0; c < chunks; c++) {
    float* nc = nm + c * stride;
    uint8_t* row = sa + (d >> 6) * ST_BLOCK + (d & 7) * 2;
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
      const int j = j0 + e;
      uint32_t q[3];
      split_pair(own[e], own[e + 1], q[0], q[1], q[2]);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        *(uint16_t*)(row + k * ST_PLANE + j * 128 + ((((d >> 3) & 7) ^ (j & 7)) << 4)) = (uint16_t)q[k];
        *(uint16_t*)(row + k * ST_PLANE + (j + 1) * 128 + ((((d >> 3) & 7) ^ ((j + 1) & 7)) << 4)) = (uint16_t)(q[k] >> 16);
      }
    }
    u.ready();
    if (tid < 32) {
      const bool one = elect_one();
      if (!mbar_wait(full + 8 * (c & 1), (c >> 1) & 1, u.abort)) u.ok = false;
      const uint32_t m = smem_u32(ma + (c & 1) * TILE_BYTES), s = smem_u32(sa);
#pragma unroll
      for (int t = 0; t < 6; t++) {
        const uint32_t pa = m + (TERM_A >> 2 * t & 3) * PLANE_BYTES, pb = s + (TERM_B >> 2 * t & 3) * ST_PLANE;
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (one) umma_bf16(u.tmem, desc_cols(pa, k), umma_desc_sw128(pb + (k >> 2) * ST_BLOCK + (k & 3) * 32), id, (t | k) ? 1u : 0u);
      }
      u.commit();
    }
    float4 next[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      next[e] = c + 1 < chunks ? *(const float4*)(nc + stride + e * Q * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      *(float4*)(nc + e * Q * 4) = make_float4(own[4 * e], own[4 * e + 1], own[4 * e + 2], own[4 * e + 3]);      // the state in front of the chunk
    }
    u.done();
    if (tid == 0 && c + 2 < chunks && u.ok) {
      fetch_m(c + 2);
      fetched = c + 3;
    }
    uint32_t w[16];
    tmem_ld16(u.tmem + ((uint32_t)((warp & 3) * 32) << 16) + j0, w);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int e = 0; e < 4; e++) {
      own[4 * e] = __uint_as_float(w[4 * e]) + add[e].x;
      own[4 * e + 1] = __uint_as_float(w[4 * e + 1]) + add[e].y;
      own[4 * e + 2] = __uint_as_float(w[4 * e + 2]) + add[e].z;
      own[4 * e + 3] = __uint_as_float(w[4 * e + 3]) + add[e].w;
      add[e] = next[e];
    }
  }
  if (tid == 0 && !u.ok) {                           // a wait was given up: let the copies that are under way land
    volatile int never = 0;
    for (int c = max(0, fetched - 2); c < fetched; c++) mbar_wait(full + 8 * (c & 1), (c >> 1) & 1, &never);
  }
#pragma unroll
  for (int e = 0; e < 16; e++)
    if (d < p.dk && v0 + e < p.dv) st[e] = own[e];
  u.close(p.err);
}

template <bool VEC>
__global__ void __launch_bounds__(NT, 1) chunk_delta_out_kernel(DeltaArgs p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int b = blockIdx.z, start = p.seq_start[b], len = p.seq_start[b + 1] - start, r0 = blockIdx.x * Q;
  if (r0 >= len) return;
  uint8_t* xa = aligned_smem(smem_raw);
  uint8_t* ya = xa + TILE_BYTES;
  const int n = min(Q, len - r0), h = p.h0 + blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t mat = ((first_chunk(start, b) + blockIdx.x) * p.hs + blockIdx.y) * MAT;
  float fq[PIECES][8], fs[PIECES][8];
  fetch_quads(fq, p.qp + mat);
  fetch_quads(fs, p.n + mat);
  Unit u;
  u.open(ya + TILE_BYTES);
  pdl_launch_dependents();               // (behind the allocation: a dependent's block must not take the columns first)
  put_quads(xa, fq);
  put_quads(ya, fs);
  u.ready();
  if (threadIdx.x < 32) {
    product<false, true>(u.tmem, smem_u32(xa), smem_u32(ya), (p.dk + 15) / 16);
    u.commit();
  }
  const int i = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
  float4 f[8];
#pragma unroll
  for (int k = 0; k < 8; k++) f[k] = *(const float4*)(p.o0 + mat + quad(i, c0 + 4 * k));
  u.done();
  uint32_t w[32];
  take(u.tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0, w);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    w[4 * k] = __float_as_uint(__uint_as_float(w[4 * k]) + f[k].x);
    w[4 * k + 1] = __float_as_uint(__uint_as_float(w[4 * k + 1]) + f[k].y);
    w[4 * k + 2] = __float_as_uint(__uint_as_float(w[4 * k + 2]) + f[k].z);
    w[4 * k + 3] = __float_as_uint(__uint_as_float(w[4 * k + 3]) + f[k].w);
  }
  float* t = (float*)xa;
  stage_lane(t, i, c0, w);
  __syncthreads();
  write_rows<VEC>(t, p.o + ((size_t)(start + r0) * p.H + h) * p.dv, (size_t)p.H * p.dv, n, p.dv);
  u.close(p.err);
}

template <typename K>
static cudaError_t allow_smem(K kernel, size_t smem) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

}  // namespace chunked

// proj [T, ld]: raw q, k, v of the heads from columns q_col, k_col, v_col; decay float [H]; state float [slots][H][D][V], read and
// advanced; chunk_state float [T / 128 + n_seqs][heads_held][D][V]: heads_held heads are gone through at a time; o float [T, H V]; err
// int or null.
SLLM_EXPORT int sllm_chunk_lin_attn_bf16(const void* proj, int ld, int q_col, int k_col, int v_col, const float* decay, float* state,
                                         const int* seq_start, const int* slots, float* chunk_state, int heads_held, float* o, int n_seqs,
                                         int max_new, int H, int D, int V, int* err, cudaStream_t stream) {
  if (n_seqs <= 0 || max_new <= 0) return 0;
  const int vblocks = (V + chunked::Q - 1) / chunked::Q;
  if (H < 1 || heads_held < 1 || D < 1 || D > chunked::Q || V < 1 || n_seqs > 65535 || (long long)H * vblocks > 65535) return SLLM_ERR_ARG;
  const int vec = !((ld | q_col | k_col | v_col | D | V) & 7) && !(((uintptr_t)proj | (uintptr_t)state | (uintptr_t)chunk_state | (uintptr_t)o) & 15);
  cudaError_t e = chunked::allow_smem(chunked::chunk_lin_states_kernel, chunked::LIN_SMEM);
  if (e == cudaSuccess) e = chunked::allow_smem(chunked::chunk_lin_scan_kernel, chunked::LIN_SMEM);
  if (e != cudaSuccess) return (int)e;
  const int chunks = (max_new + chunked::Q - 1) / chunked::Q, DV = D * V;
  for (int h0 = 0; h0 < H; h0 += heads_held) {
    const int hs = H - h0 < heads_held ? H - h0 : heads_held;
    chunked::LinArgs p{(const bf16*)proj, ld, q_col, k_col, v_col, decay, state, seq_start, slots, chunk_state, o, H, D, V, h0, hs, err, vec};
    const dim3 grid(chunks, hs * vblocks, n_seqs);
    sllm_launch(chunked::chunk_lin_states_kernel, grid, dim3(chunked::NT), chunked::LIN_SMEM, stream, p);
    if (vec) sllm_launch(chunked::chunk_lin_pass_kernel<4>, dim3((DV / 4 + 255) / 256, hs, n_seqs), dim3(256), 0, stream, p);
    else sllm_launch(chunked::chunk_lin_pass_kernel<1>, dim3((DV + 255) / 256, hs, n_seqs), dim3(256), 0, stream, p);
    sllm_launch(chunked::chunk_lin_scan_kernel, grid, dim3(chunked::NT), chunked::LIN_SMEM, stream, p);
  }
  SLLM_RETURN_LAST();
}

// qk float rows [G dk | G dk], v float rows [H dv], bd float [T, 2 H + G] as the walk takes them; state float [slots][H][dk][dv], read
// and advanced; scratch: sllm_chunk_delta_scratch() bytes for each of `heads_held` heads (gone through that many at a time) of each of
// `chunks_held` >= T / 128 + n_seqs chunks, 16-byte aligned; o float [T, H dv]; dk and dv up to 128.
SLLM_EXPORT int sllm_chunk_delta_scratch(void) { return (int)(chunked::TILE_BYTES + 3 * chunked::MAT * sizeof(float)); }
SLLM_EXPORT int sllm_chunk_delta(const float* qk, int ld_qk, const float* v, int ld_v, const float* bd, float* state, const int* seq_start,
                                 const int* slots, void* scratch, long long chunks_held, int heads_held, float* o, int n_seqs, int max_new,
                                 int H, int G, int dk, int dv, int* err, cudaStream_t stream) {
  using namespace chunked;
  if (n_seqs <= 0 || max_new <= 0) return 0;
  if (H < 1 || heads_held < 1 || G < 1 || H % G || dk < 1 || dk > Q || dv < 1 || dv > Q || n_seqs > 65535 || H > 65535 || ((uintptr_t)scratch & 15))
    return SLLM_ERR_ARG;
  const bool vec = !((ld_qk | ld_v | dk | dv) & 7) && !(((uintptr_t)qk | (uintptr_t)v | (uintptr_t)o) & 15);
  const auto parts = vec ? chunk_delta_parts_kernel<true> : chunk_delta_parts_kernel<false>;
  const auto out = vec ? chunk_delta_out_kernel<true> : chunk_delta_out_kernel<false>;
  cudaError_t e = allow_smem(parts, DELTA_SMEM);
  if (e == cudaSuccess) e = allow_smem(chunk_delta_pass_kernel, PASS_SMEM);
  if (e == cudaSuccess) e = allow_smem(out, DELTA_SMEM);
  if (e != cudaSuccess) return (int)e;
  for (int h0 = 0; h0 < H; h0 += heads_held) {
    const int hs = H - h0 < heads_held ? H - h0 : heads_held;
    const size_t units = (size_t)chunks_held * hs;
    float* mats = (float*)((uint8_t*)scratch + units * TILE_BYTES);
    DeltaArgs p{qk, ld_qk, v, ld_v, bd, state, seq_start, slots, (uint8_t*)scratch, mats, mats + units * MAT, mats + 2 * units * MAT, o, H, G, dk, dv,
                h0, hs, err};
    const dim3 grid((max_new + Q - 1) / Q, hs, n_seqs);
    sllm_launch(parts, grid, dim3(NT), DELTA_SMEM, stream, p);
    sllm_launch(chunk_delta_pass_kernel, dim3((dv + PV - 1) / PV, hs, n_seqs), dim3(256), PASS_SMEM, stream, p);
    sllm_launch(out, grid, dim3(NT), DELTA_SMEM, stream, p);
  }
  SLLM_RETURN_LAST();
}
