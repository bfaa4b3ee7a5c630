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
#include "split_mma.cuh"

namespace chunked {
using namespace sm3;

constexpr int Q = TILE, NT = 512, PIECES = Q * Q / 8 / NT;      // rows of a chunk, threads, 8-column pieces of a tile a thread makes

// z / (1 + exp(-z)); the reciprocal is the hardware's with one Newton step (its error is then a float's last place), and the
// exponential is held below where that step would meet an infinity
__device__ __forceinline__ float silu_f(float z) {
  const float d = 1.0f + fminf(expf(-z), 1e36f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return z * fmaf(r, fmaf(-d, r, 1.0f), r);
}

struct LinArgs {
  const bf16* proj; int ld, q_col, k_col, v_col;      // raw projections, one row a token
  const float* decay;                                 // [H]
  float* state;                                       // [slots][H][D][V]
  const int* seq_start; const int* slots;
  float* chunk_state;                                 // [chunks][H][D][V]
  float* o;                                           // [T][H V]
  int H, D, V;
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
// silu of what was fetched, row r times scale[r] (null: 1), into the tile's planes
__device__ __forceinline__ void put_silu(uint8_t* tile, const uint4 (&raw)[PIECES], const float* scale) {
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
  extern __shared__ uint8_t smem_raw[];
  const int b = blockIdx.z, start = p.seq_start[b], len = p.seq_start[b + 1] - start, r0 = blockIdx.x * Q;
  if (r0 >= len) return;
  uint8_t* ka = aligned_smem(smem_raw);
  uint8_t* va = ka + TILE_BYTES;
  float* pw = (float*)(va + TILE_BYTES);
  float* scale = pw + Q + 4;
  const int n = min(Q, len - r0), vblocks = (p.V + Q - 1) / Q, h = blockIdx.y / vblocks, v0 = (blockIdx.y % vblocks) * Q;
  const int vn = min(Q, p.V - v0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bf16* row = p.proj + (size_t)(start + r0) * p.ld;
  uint4 kr[PIECES], vr[PIECES];
  fetch(kr, row + p.k_col + (size_t)h * p.D, p.ld, n, p.D, p.vec);
  fetch(vr, row + p.v_col + (size_t)h * p.V + v0, p.ld, n, vn, p.vec);
  fill_powers(pw, p.decay[h]);
  Unit u;
  u.open((uint8_t*)(scale + Q + 4));
  if (tid < Q) scale[tid] = tid < n ? pw[n - 1 - tid] : 0.f;
  put_silu(va, vr, nullptr);
  __syncthreads();
  put_silu(ka, kr, scale);
  u.ready();
  if (tid == 0) {
    product<true, true>(u.tmem, smem_u32(ka), smem_u32(va), (n + 15) / 16);
    u.commit();
  }
  u.done();
  const int d = (warp & 3) * 32 + lane;
  float* dst = p.chunk_state + (((first_chunk(start, b) + blockIdx.x) * p.H + h) * p.D + d) * (size_t)p.V + v0;
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
  const int b = blockIdx.z, h = blockIdx.y, start = p.seq_start[b], len = p.seq_start[b + 1] - start;
  const int DV = p.D * p.V, e0 = (blockIdx.x * 256 + threadIdx.x) * E;
  if (e0 >= DV || len <= 0) return;
  const int chunks = (len + Q - 1) / Q;
  const size_t stride = (size_t)p.H * DV;
  float* u = p.chunk_state + (first_chunk(start, b) * p.H + h) * (size_t)DV + e0;
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
  extern __shared__ uint8_t smem_raw[];
  const int b = blockIdx.z, start = p.seq_start[b], len = p.seq_start[b + 1] - start, r0 = blockIdx.x * Q;
  if (r0 >= len) return;
  uint8_t* qa = aligned_smem(smem_raw);
  uint8_t* xa = qa + TILE_BYTES;                   // the state, then the keys, then the values
  float* pw = (float*)(xa + TILE_BYTES);
  const int n = min(Q, len - r0), vblocks = (p.V + Q - 1) / Q, h = blockIdx.y / vblocks, v0 = (blockIdx.y % vblocks) * Q;
  const int vn = min(Q, p.V - v0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bf16* row = p.proj + (size_t)(start + r0) * p.ld;
  uint4 raw[PIECES];
  fetch(raw, row + p.q_col + (size_t)h * p.D, p.ld, n, p.D, p.vec);
  fill_powers(pw, p.decay[h]);
  Unit u;
  u.open((uint8_t*)(pw + 2 * (Q + 4)));
  put_silu(qa, raw, nullptr);
  put_floats(xa, p.chunk_state + ((first_chunk(start, b) + blockIdx.x) * p.H + h) * (size_t)p.D * p.V + v0, p.V, p.D, vn, p.vec);
  u.ready();
  const int dsteps = (p.D + 15) / 16, rsteps = (n + 15) / 16;
  if (tid == 0) {
    product<false, true>(u.tmem, smem_u32(qa), smem_u32(xa), dsteps);
    u.commit();
  }
  fetch(raw, row + p.k_col + (size_t)h * p.D, p.ld, n, p.D, p.vec);
  u.done();
  put_silu(xa, raw, nullptr);
  u.ready();
  if (tid == 0) {
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
    put_silu(xa, raw, nullptr);                    // the keys have been read
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
  if (tid == 0) {
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
  if (i < n) store_row(dst, c, c0, vn, p.vec);
  u.close(p.err);
}

template <typename K>
static cudaError_t allow_smem(K kernel, size_t smem) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

}  // namespace chunked

// proj [T, ld]: raw q, k, v of the heads from columns q_col, k_col, v_col; decay float [H]; state float [slots][H][D][V], read and
// advanced; chunk_state float [T / 128 + n_seqs][H][D][V]; o float [T, H V]; err int or null.
SLLM_EXPORT int sllm_chunk_lin_attn_bf16(const void* proj, int ld, int q_col, int k_col, int v_col, const float* decay, float* state,
                                         const int* seq_start, const int* slots, float* chunk_state, float* o, int n_seqs, int max_new,
                                         int H, int D, int V, int* err, cudaStream_t stream) {
  if (n_seqs <= 0 || max_new <= 0) return 0;
  const int vblocks = (V + chunked::Q - 1) / chunked::Q;
  if (H < 1 || D < 1 || D > chunked::Q || V < 1 || n_seqs > 65535 || (long long)H * vblocks > 65535) return SLLM_ERR_ARG;
  const int vec = !((ld | q_col | k_col | v_col | D | V) & 7) && !(((uintptr_t)proj | (uintptr_t)state | (uintptr_t)chunk_state | (uintptr_t)o) & 15);
  chunked::LinArgs p{(const bf16*)proj, ld, q_col, k_col, v_col, decay, state, seq_start, slots, chunk_state, o, H, D, V, err, vec};
  cudaError_t e = chunked::allow_smem(chunked::chunk_lin_states_kernel, chunked::LIN_SMEM);
  if (e == cudaSuccess) e = chunked::allow_smem(chunked::chunk_lin_scan_kernel, chunked::LIN_SMEM);
  if (e != cudaSuccess) return (int)e;
  const int chunks = (max_new + chunked::Q - 1) / chunked::Q, DV = D * V;
  const dim3 grid(chunks, H * vblocks, n_seqs);
  chunked::chunk_lin_states_kernel<<<grid, chunked::NT, chunked::LIN_SMEM, stream>>>(p);
  if (vec) chunked::chunk_lin_pass_kernel<4><<<dim3((DV / 4 + 255) / 256, H, n_seqs), 256, 0, stream>>>(p);
  else chunked::chunk_lin_pass_kernel<1><<<dim3((DV + 255) / 256, H, n_seqs), 256, 0, stream>>>(p);
  chunked::chunk_lin_scan_kernel<<<grid, chunked::NT, chunked::LIN_SMEM, stream>>>(p);
  SLLM_RETURN_LAST();
}
