// Products of float matrices on the 5th-generation tensor cores: C[M,N] = A[M,K] * B[N,K]^T.
//
// A float of 2^-110 or more is the sum of three bfloat16 numbers (see split_mma.cuh: 8 + 8 + 8 bits); below, its last bits lie under
// the smallest bfloat16. So a first kernel writes both operands times 2^24 as three planes of bfloat16: exact for every float up to
// 2^104, subnormal ones included. A second one multiplies the planes: the six largest terms (2,0) (0,2) (1,1) (1,0) (0,1) (0,0) of a
// product of two such sums, smallest first; what is left out comes to 2^-24 of the product at most. Results are scaled back by 2^-48; what
// overflows under way, a float above 2^104 or a sum of 2^80 or more, goes the way of what is not finite (below).
//
// Sums in tensor memory cut what does not fit their 24 bits at every step, which a long sum cannot afford (8,192 terms in one
// accumulator: 9.1e-6 off, a chain of FMA 1.6e-6). So a sum ends after 64 terms of K: the epilogue's warps keep the tile's outputs as
// floats in registers and add each finished accumulator to them, rounding to nearest, while the other accumulator of the two is filled.
//
// Bound by the tensor cores: six products for one. Two SMs share a tile of 256 x BN (as gemm_tc_pair_kernel in gemm_tcgen05.cu), a
// k-block of 64 is 96 KB of planes an SM, and the ring holds two. Its three parts (second rests, first rests, heads) are handed back one
// by one as the six terms run, so the copies of the block after next start a third, five sixths and all of a block's time ahead.
//
// Measured, FMA kernels / here with the planes' kernel, us: 2,778 rows by 2,560 x 1,024 285 / 76, by five blocks of 512 x 256 77 / 31;
// 4,096 rows by 8,192 x 2,048 2,590 / 560 (1,475 TFLOP/s of products). Errors (2-norm, against 64 bits) of normal operands, 1,024 terms
// 5.7e-7 / 1.1e-7, 8,192 1.6e-6 / 2.2e-7, 64 1.4e-7 / 7.8e-8; of positive ones 4.9e-7 / 1.1e-7, 1.4e-6 / 2.0e-7, 1.2e-7 / 9.2e-8.
// The exception is a sum that one term makes up: cut in tensor memory it is 5e-8 off (rms), rounded once by a chain 2.5e-8.
//
// What is not finite comes out not finite of any term it meets (a head that rounds up to infinity included), so an output that is not
// finite is computed again by its chain of FMA, from the floats: by the warp that stored it, when its tiles are done and nothing waits
// for it, rows that hold one eight at a time. 1,000 rows by 2,560 x 2,048 84 us, with a row of NaN 246, all NaN 1,950 (FMA kernel 393; an
// output a thread at a time, in front of waiting tiles: the one row 5,665).
#include "tcgen05.cuh"

#define GS_BK 64
#define GS_BM 256
#define GS_THREADS 320            // a warp of copies, a warp of products, eight of sums
#define GS_SCALE 0x1p24f          // of either operand in its planes
#define GS_SLOTS 6                // three parts of a k-block, two k-blocks

// One operand's floats as three planes [3][rows][cols] of bfloat16, eight elements a thread; both operands in one launch (blockIdx.y).
struct GsSplit { const float* src; bf16* dst; int rows, cols, ld; };
__global__ void __launch_bounds__(256) gemm_split_planes_kernel(const GsSplit sa, const GsSplit sb) {
  pdl_launch_dependents();
  pdl_wait();
  const GsSplit s = blockIdx.y ? sb : sa;
  const int groups = s.cols >> 3;
  const long long total = (long long)s.rows * groups, plane = (long long)s.rows * s.cols;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int row = (int)(i / groups), c = (int)(i - (long long)row * groups) << 3;
    F8 f = ld8(s.src + (size_t)row * s.ld + c);
#pragma unroll
    for (int e = 0; e < 8; e++) f.f[e] *= GS_SCALE;
    uint4 q[3];
    split_pair(f.f[0], f.f[1], q[0].x, q[1].x, q[2].x);
    split_pair(f.f[2], f.f[3], q[0].y, q[1].y, q[2].y);
    split_pair(f.f[4], f.f[5], q[0].z, q[1].z, q[2].z);
    split_pair(f.f[6], f.f[7], q[0].w, q[1].w, q[2].w);
    bf16* d = s.dst + (size_t)row * s.cols + c;
#pragma unroll
    for (int p = 0; p < 3; p++) *(uint4*)(d + p * plane) = q[p];
  }
}

// A product, or one of `parts` along K (C receives partial sums c_part apart), or `batch` products side by side: the z-th on columns
// z * K of A, rows z * N of B, and C + z * c_part.
struct GsArgs {
  const float* a;      // the floats themselves, for outputs that come out not finite
  const float* b;
  float* c;
  int M, N, K, lda, ldb, ldc;
  int parts, batch, kb_part;       // kb_part: k-blocks to a part
  long long c_part;
  int b_rows;                      // rows of a plane of B
};

// The outputs of a warp's 32 rows and OWN columns that are not finite, by their chains of multiply-adds from k0 to k1 (in multiples of
// 8). A lane takes every 32nd column, ROWS of the rows marked in `rows` at a time, so that a column's weights are read once for them.
template <int OWN, int ROWS>
__device__ __forceinline__ void gs_rows_again(const float* a, int lda, const float* b, int ldb, float* c, int ldc, int n, uint32_t rows, int k0, int k1) {
  constexpr int COLS = OWN / 32;
  const int lane = threadIdx.x & 31;
  const float* bc[COLS];
#pragma unroll
  for (int i = 0; i < COLS; i++) bc[i] = b + (size_t)min(lane + 32 * i, n - 1) * ldb;
  while (rows) {
    const float* ar[ROWS];
    float* cr[ROWS];
    float s[ROWS][COLS];
    int r = 0, there = 0;
#pragma unroll
    for (int u = 0; u < ROWS; u++) {          // (past the last marked row: that row again, not written)
      if (rows) { r = __ffs(rows) - 1; there++; }
      rows &= rows - 1;
      ar[u] = a + (size_t)r * lda;
      cr[u] = c + (size_t)r * ldc;
#pragma unroll
      for (int i = 0; i < COLS; i++) s[u][i] = 0.f;
    }
#pragma unroll 2
    for (int k = k0; k < k1; k += 4) {
      float4 w[COLS];
#pragma unroll
      for (int i = 0; i < COLS; i++) w[i] = *(const float4*)(bc[i] + k);
#pragma unroll
      for (int u = 0; u < ROWS; u++) {
        const float4 x = *(const float4*)(ar[u] + k);
#pragma unroll
        for (int i = 0; i < COLS; i++) s[u][i] = fmaf(x.w, w[i].w, fmaf(x.z, w[i].z, fmaf(x.y, w[i].y, fmaf(x.x, w[i].x, s[u][i]))));
      }
    }
#pragma unroll
    for (int u = 0; u < ROWS; u++)
#pragma unroll
      for (int i = 0; i < COLS; i++) {
        const int col = lane + 32 * i;
        if (u < there && col < n && !(fabsf(cr[u][col]) <= 3.402823466e+38f)) cr[u][col] = s[u][i];
      }
  }
}

// Tile number: z slowest, then columns, rows fastest (tiles that run side by side share B). k-blocks kb0 .. kb0 + nkb - 1
template <int BN>
__device__ __forceinline__ void gs_tile(const GsArgs& g, int tile, int& z, int& m0, int& n0, int& kb0, int& nkb) {
  const int tiles_m = (g.M + GS_BM - 1) / GS_BM, per_z = tiles_m * ((g.N + BN - 1) / BN);
  z = tile / per_z;
  const int r = tile - z * per_z;
  m0 = (r % tiles_m) * GS_BM;
  n0 = (r / tiles_m) * BN;
  kb0 = g.batch > 1 ? 0 : z * g.kb_part;
  nkb = max(0, min(g.kb_part, (g.K + GS_BK - 1) / GS_BK - kb0));
}

// Behind a warp's last tile (its first row and column of a tile at `dm`, `dn`): the tiles in which it stored something not finite, the
// i-th if bit i % 32 of `marked` says so.
template <int BN>
__device__ __noinline__ void gs_again(const GsArgs& g, int tile, int n_pairs, int n_tiles, int dm, int dn, uint32_t marked) {
  constexpr int OWN = BN / 2;
  const int lane = threadIdx.x & 31;
  __syncwarp();
  for (int i = 0; tile < n_tiles; tile += n_pairs, i++) {
    if (!(marked >> (i & 31) & 1)) continue;
    int z, m0, n0, kb0, nkb;
    gs_tile<BN>(g, tile, z, m0, n0, kb0, nkb);
    const int row0 = m0 + dm, col = n0 + dn, n = min(OWN, g.N - col), k0 = kb0 * GS_BK, k1 = min(g.K, (kb0 + nkb) * GS_BK);
    float* c = g.c + (g.parts > 1 || g.batch > 1 ? z * g.c_part : 0) + (size_t)row0 * g.ldc + col;
    bool bad = false;
    if (row0 + lane < g.M)
      for (int j = 0; j < n; j++) bad |= !(fabsf(c[(size_t)lane * g.ldc + j]) <= 3.402823466e+38f);
    const uint32_t rows = __ballot_sync(0xffffffffu, bad);
    if (!rows) continue;
    const float* a = g.a + (size_t)row0 * g.lda + (g.batch > 1 ? (size_t)z * g.K : 0);
    const float* b = g.b + ((g.batch > 1 ? (size_t)z * g.N : 0) + col) * g.ldb;
    if (__popc(rows) > 1) gs_rows_again<OWN, 8>(a, g.lda, b, g.ldb, c, g.ldc, n, rows, k0, k1);
    else gs_rows_again<OWN, 1>(a, g.lda, b, g.ldb, c, g.ldc, n, rows, k0, k1);
  }
}

__device__ __forceinline__ void gs_store8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GS_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ GsArgs g,
                  int* __restrict__ err) {
  constexpr uint32_t A_BYTES = 128 * GS_BK * 2, B_BYTES = (BN / 2) * GS_BK * 2, SLOT_BYTES = A_BYTES + B_BYTES;
  constexpr int OWN = BN / 2;                                   // columns of an epilogue warp
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + GS_SLOTS * SLOT_BYTES);   // full[SLOTS], empty[SLOTS], acc_full[2], acc_empty[2]
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * GS_SLOTS + 4);
  volatile int* abort = (volatile int*)(tmem_slot + 1);
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * GS_SLOTS, acc_full0 = empty0 + 8 * GS_SLOTS, acc_empty0 = acc_full0 + 16;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int n_tiles = (g.M + GS_BM - 1) / GS_BM * ((g.N + BN - 1) / BN) * g.parts * g.batch;

  if (threadIdx.x == 0) {
    for (int s = 0; s < GS_SLOTS; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    for (int a = 0; a < 2; a++) { mbar_init(acc_full0 + 8 * a, 1); mbar_init(acc_empty0 + 8 * a, 16); }
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if (lane == 0) *tmem_slot = 0;
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();                   // the other block's barriers are set up before anything arrives on them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();               // (behind the allocation: a dependent's block must not take the columns first)
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int it = 0, issued = 0;           // k-blocks begun; slots filled so far (three a k-block)
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
        int z, m0, n0, kb0, nkb;
        gs_tile<BN>(g, tile, z, m0, n0, kb0, nkb);
        const int am = m0 + (int)rank * 128, bn = (g.batch > 1 ? z * g.N : 0) + n0 + (int)rank * (BN / 2), ak = g.batch > 1 ? z * g.K : 0;
        for (int kb = 0; kb < nkb && ok; kb++, it++) {
          for (int part = 0; part < 3; part++) {                // plane 2 - part of both operands into slot 2 part + (it & 1)
            const int s = 2 * part + (it & 1), plane = 2 - part;
            ok = mbar_wait(empty0 + 8 * s, ((it >> 1) & 1) ^ 1, abort);
            if (!ok) break;
            if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * SLOT_BYTES);      // both blocks' bytes
            const uint32_t full_lead = mapa_shared(full0 + 8 * s, 0), dst = smem_base + s * SLOT_BYTES;
            tma_load_2d_pair(dst, &map_a, ak + (kb0 + kb) * GS_BK, plane * g.M + am, full_lead);
            tma_load_2d_pair(dst + A_BYTES, &map_b, (kb0 + kb) * GS_BK, plane * g.b_rows + bn, full_lead);
            issued++;
          }
        }
      }
      if (*abort) {
        // copies already issued still land in this block's shared memory. Rank 0 sees them on its own barriers; the other
        // block cannot wait on those and gives its copies ample time instead.
        if (rank == 0) {
          volatile int never = 0;
          for (int j = max(0, issued - GS_SLOTS); j < issued; j++) {
            const int i = j / 3, s = 2 * (j % 3) + (i & 1);
            mbar_wait(full0 + 8 * s, (i >> 1) & 1, &never);
          }
        } else {
          uint64_t t0 = global_ns();
          while (global_ns() - t0 < 1000000ull) __nanosleep(1000);
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      const bool one = elect_one();
      constexpr uint32_t idesc = umma_idesc_bf16(GS_BM, BN);
      int it = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
        int z, m0, n0, kb0, nkb;
        gs_tile<BN>(g, tile, z, m0, n0, kb0, nkb);
        for (int kb = 0; kb < nkb; kb++, it++) {
          const int a = it & 1;
          const uint32_t ph = (it >> 1) & 1, acc = tmem_base + (uint32_t)(a * BN);
          const uint32_t s2 = a, s1 = 2 + a, s0 = 4 + a;        // the slots of planes 2, 1, 0
          auto term = [&](uint32_t sa, uint32_t sb, bool first) {
            const uint32_t a_addr = smem_base + sa * SLOT_BYTES, b_addr = smem_base + sb * SLOT_BYTES + A_BYTES;
#pragma unroll
            for (int k = 0; k < GS_BK / 16; k++)
              if (one) umma_bf16_pair(acc, umma_desc_sw128(a_addr + k * 32), umma_desc_sw128(b_addr + k * 32), idesc, (first && k == 0) ? 0u : 1u);
          };
          ok = mbar_wait_cluster(acc_empty0 + 8 * a, ph ^ 1, abort)        // both blocks have taken this accumulator's last sums
               && mbar_wait(full0 + 8 * s2, ph, abort) && mbar_wait(full0 + 8 * s0, ph, abort);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          term(s2, s0, true);
          term(s0, s2, false);
          if (one) umma_commit_pair(empty0 + 8 * s2);
          ok = mbar_wait(full0 + 8 * s1, ph, abort);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          term(s1, s1, false);
          term(s1, s0, false);
          term(s0, s1, false);
          if (one) umma_commit_pair(empty0 + 8 * s1);
          term(s0, s0, false);
          if (one) {
            umma_commit_pair(empty0 + 8 * s0);
            umma_commit_pair(acc_full0 + 8 * a);
          }
        }
      }
    }
  } else {
    const int q = warp & 3, c_lo = warp < 6 ? 0 : OWN;
    const uint32_t trow = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c_lo;
    int it = 0, i = 0;
    uint32_t marked = 0;                // of the tiles, by their number modulo 32: something not finite was stored
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, i++) {
      int z, m0, n0, kb0, nkb;
      gs_tile<BN>(g, tile, z, m0, n0, kb0, nkb);
      float sum[OWN];
#pragma unroll
      for (int j = 0; j < OWN; j++) sum[j] = 0.f;
      for (int kb = 0; kb < nkb; kb++, it++) {
        const int a = it & 1;
        ok = mbar_wait(acc_full0 + 8 * a, (it >> 1) & 1, abort);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < OWN; c += 16) {
          uint32_t r[16];
          tmem_ld16(trow + (uint32_t)(a * BN + c), r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; j++) sum[c + j] += __uint_as_float(r[j]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_shared(acc_empty0 + 8 * a, 0));
      }
      if (!ok) break;
#pragma unroll
      for (int j = 0; j < OWN; j++) sum[j] *= 1.0f / (GS_SCALE * GS_SCALE);
      const int row = m0 + (int)rank * 128 + q * 32 + lane, col = n0 + c_lo;
      bool bad = false;
      if (row < g.M && col < g.N) {
        float* dst = g.c + (g.parts > 1 || g.batch > 1 ? z * g.c_part : 0) + (size_t)row * g.ldc + col;
        const bool vec = ((uintptr_t)dst & 31) == 0;
#pragma unroll
        for (int j = 0; j < OWN; j += 8) {
          if (vec && col + j + 8 <= g.N) {
            gs_store8(dst + j, sum + j);
          } else {
#pragma unroll
            for (int e = 0; e < 8; e++)
              if (col + j + e < g.N) dst[j + e] = sum[j + e];
          }
#pragma unroll
          for (int e = 0; e < 8; e++) bad |= !(fabsf(sum[j + e]) <= 3.402823466e+38f);
        }
      }
      if (__any_sync(0xffffffffu, bad)) marked |= 1u << (i & 31);
    }
    if (ok && marked) gs_again<BN>(g, pair, n_pairs, n_tiles, (int)rank * 128 + q * 32, c_lo, marked);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();                   // nothing of the other block is still on its way to this one
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * BN) : "memory");
  }
  if (threadIdx.x == 0 && *abort && err) atomicExch(err, 2);
}

// ------------------------------------------------------------------ host side
template <int BN>
static int gs_launch(const CUtensorMap& ma, const CUtensorMap& mb, const GsArgs& g, int* err, cudaStream_t stream) {
  constexpr size_t smem = GS_SLOTS * (128 + BN / 2) * GS_BK * 2 + 1024 + 256;
  static SllmPerDevice held;             // how many pairs of blocks the GPU holds at once
  std::atomic<int>& pairs = held.here();
  if (!pairs.load()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int sms = sllm_sm_count();
    if (sms < 2) return SLLM_ERR_ARG - 3;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms & ~1);
    cfg.blockDim = dim3(GS_THREADS);
    cfg.dynamicSmemBytes = smem;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_split_kernel<BN>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = sms / 2;
    }
    pairs.store(n < sms / 2 ? n : sms / 2);
  }
  const long long tiles = (long long)((g.N + BN - 1) / BN) * ((g.M + GS_BM - 1) / GS_BM) * g.parts * g.batch;
  if (tiles > 0x7fffffffLL) return SLLM_ERR_ARG;
  const dim3 grid(2 * (int)(tiles < pairs.load() ? tiles : pairs.load()));
  sllm_launch(gemm_split_kernel<BN>, grid, dim3(GS_THREADS), smem, stream, ma, mb, g, err);
  SLLM_RETURN_LAST();
}

static int gs_product(const GsArgs& g, const bf16* planes_a, const bf16* planes_b, int tile_n, int* err, cudaStream_t stream) {
  const int a_cols = g.batch * g.K;
  CUtensorMap ma, mb;
  int rc = tc_make_map(&ma, planes_a, 3 * g.M, a_cols, a_cols, 128);
  if (!rc) rc = tc_make_map(&mb, planes_b, 3 * g.b_rows, g.K, g.K, tile_n / 2);
  if (rc) return rc;
  return tile_n == 256 ? gs_launch<256>(ma, mb, g, err, stream) : gs_launch<128>(ma, mb, g, err, stream);
}

// Columns of a tile: 128 where the tiles of 256 leave more of the last wave of pairs idle than narrow tiles, which read A's planes
// twice as often, lose.
static int gs_tile_n(int M, int N, int z) {
  const long long rows = (M + GS_BM - 1) / GS_BM * (long long)z, wide = rows * ((N + 255) / 256), narrow = rows * ((N + 127) / 128);
  const int pairs = sllm_sm_count() / 2 > 0 ? sllm_sm_count() / 2 : 1;
  return (narrow + pairs - 1) / pairs * 11 < (wide + pairs - 1) / pairs * 20 ? 128 : 256;
}

// C[M,N] = A[M,K] B[N,K]^T, floats. parts > 1: K is cut into that many runs and C receives their partial sums, c_part apart. batch > 1:
// products side by side, the z-th of A's columns z K .. with B's rows z N .. into C + z c_part (parts 1). `scratch` receives the planes;
// where it is smaller than the 6 (M batch + N batch) K bytes of both, rows and columns go in portions that fit, one after the other.
// K and the row strides in multiples of 8 / 4 elements, 16-byte aligned operands. *err (or null) is set to 2 if a wait runs out of time.
SLLM_EXPORT int sllm_gemm_split_f32(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc, int parts,
                                    int batch, long long c_part, void* scratch, long long scratch_bytes, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (K <= 0 || (K & 7) || (lda & 3) || (ldb & 3) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15) || ((uintptr_t)C & 3) || parts < 1 ||
      (parts > 1 && batch > 1) || !scratch || ((uintptr_t)scratch & 15))
    return SLLM_ERR_ARG;
  const long long a_row = 6ll * K * batch, b_row = 6ll * K * batch;          // bytes of planes to a row of A, to a column of C (all of the batch's)
  if ((long long)batch * K > 0x7fffffffLL || (long long)batch * N * 3 > 0x7fffffffLL) return SLLM_ERR_ARG;
  long long mp = M, np = N;
  if (M * a_row + N * b_row > scratch_bytes) {
    const long long half = scratch_bytes / 2;
    if (N * b_row <= half) mp = (scratch_bytes - N * b_row) / a_row;
    else if (M * a_row <= half) np = (scratch_bytes - M * a_row) / b_row;
    else { mp = half / a_row; np = half / b_row; }
    if (mp < M) mp = mp / GS_BM * GS_BM;
    if (np < N) np = np / 256 * 256;
    if (mp < 1 || np < 1 || (batch > 1 && np < N)) return SLLM_ERR_ARG;      // (a batch's columns are not cut)
  }
  const int nkb = (K + GS_BK - 1) / GS_BK, kb_part = (nkb + parts - 1) / parts, at_once = sllm_sm_count() * 8;
  bf16* pa = (bf16*)scratch;
  bf16* pb = (bf16*)((char*)scratch + mp * a_row);
  for (long long n0 = 0; n0 < N; n0 += np) {
    const int n = (int)(N - n0 < np ? N - n0 : np);
    for (long long m0 = 0; m0 < M; m0 += mp) {
      const int m = (int)(M - m0 < mp ? M - m0 : mp);
      GsSplit sa{A + m0 * lda, pa, m, batch * K, lda}, sb{B + n0 * ldb, pb, batch * n, K, ldb};
      if (mp >= M && n0 > 0) sa.rows = 0;          // still there
      if (m0 > 0) sb.rows = 0;
      const long long most = ((long long)(sa.rows) * sa.cols > (long long)sb.rows * K ? (long long)sa.rows * sa.cols : (long long)sb.rows * K) / 8;
      const long long blocks = (most + 255) / 256;
      sllm_launch(gemm_split_planes_kernel, dim3((unsigned)(blocks < at_once ? blocks : at_once), 2), dim3(256), 0, stream, sa, sb);
      const GsArgs g{A + m0 * lda, B + n0 * ldb, C + m0 * ldc + n0, m, n, K, lda, ldb, ldc, parts, batch, kb_part, c_part, batch * n};
      const int rc = gs_product(g, pa, pb, gs_tile_n(m, n, parts * batch), err, stream);
      if (rc) return rc;
    }
  }
  return 0;
}
