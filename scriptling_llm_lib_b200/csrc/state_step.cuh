// A decode step of a recurrence with a matrix state per head: S <- dec S + d b x^T, y = S^T c, one row a sequence.
//
// The step reads and writes every sequence's states once and does little else, so the states are moved by bulk copies: a block stays and
// walks (sequence, head) pairs; a ring of three tiles [rows][cols] in shared memory has the next pairs' states on their way in and the
// last one's on its way out while a pair's row is worked on in place (cols / 4 lanes a row of the state). What a row brings comes a
// pair ahead through registers. Bound by the copies. A job says where states lie, what a row brings and what becomes of y.
//
// A block whose wait for a pair's states runs out stores nothing of that pair or of those behind it: it lets the copies that are under
// way land, raises the error flag and leaves.
#pragma once
#include "tcgen05.cuh"

namespace step {

constexpr int RING = 3;

struct Row { float b, c, x, z, d, dec; };      // element tid of b and c (rows), of x and z (cols); d and dec of thread 0

// the widths the walk takes: a row of the state is shared out to whole parts of a warp, and the ring fits
static inline bool takes(int rows, int cols) {
  return cols >= 16 && cols <= 128 && (cols & (cols - 1)) == 0 && rows >= 1 && rows <= 256 && (size_t)rows * cols * 4 <= 64 * 1024;
}
static inline size_t smem_bytes(int rows, int cols) {
  return ((size_t)RING * rows * cols + 8 * cols + 2 * ((2 * rows + 2 * cols + 7) & ~3)) * sizeof(float) + 8 * RING + 16;
}

template <typename Job>
__global__ void __launch_bounds__(256) state_step_kernel(Job job, int units, int* err) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int N = job.rows(), V = job.cols(), H = job.heads(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t tile_bytes = (uint32_t)N * V * 4;
  float* tiles = (float*)smem_raw;                              // [ring][N][V]
  float* red = tiles + (size_t)RING * N * V;                    // [8][V]
  float* rows = red + 8 * V;                                    // two of [x: V | z: V | d, dec, -, - | b: N | c: N]
  const int row_len = (2 * N + 2 * V + 7) & ~3, at_b = 2 * V + 4;
  uint8_t* head = (uint8_t*)(rows + 2 * row_len);
  const uint32_t full = smem_u32(head);
  volatile int* abort = (volatile int*)(head + 8 * RING);
  if (tid == 0) {
    for (int s = 0; s < RING; s++) mbar_init(full + 8 * s, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int mine = ((int)blockIdx.x < units) ? (units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto pair = [&](int i, int& b, int& h) {                      // this block's i-th pair
    const int u = blockIdx.x + i * gridDim.x;
    b = u / H;
    h = u % H;
  };
  auto load = [&](int i) {
    int b, h;
    pair(i, b, h);
    const uint32_t bar = full + 8 * (i % RING);
    mbar_expect_tx(bar, tile_bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(tiles + (size_t)(i % RING) * N * V)), "l"(job.place(b, h)), "r"(tile_bytes), "r"(bar) : "memory");
  };
  if (tid == 0)
    for (int i = 0; i < min(mine, RING - 1); i++) load(i);
  Row next = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  auto fetch = [&](int i) {
    int b, h;
    pair(i, b, h);
    job.fetch(next, b, h, tid);
  };
  auto stash = [&](int i) {
    float* d = rows + (i & 1) * row_len;
    if (tid < N) { d[at_b + tid] = next.b; d[at_b + N + tid] = next.c; }
    if (tid < V) { d[tid] = next.x; d[V + tid] = next.z; }
    if (tid == 0) { d[2 * V] = next.d; d[2 * V + 1] = next.dec; }
  };
  if (mine > 0) {
    fetch(0);
    stash(0);
  }
  __syncthreads();
  const int per = V / 4, rows_at_once = 256 / per, c4 = (tid % per) * 4, r0 = tid / per;
  bool ok = true;
  for (int i = 0; i < mine; i++) {
    if (!mbar_wait(full + 8 * (i % RING), (i / RING) & 1, abort)) ok = false;
    if (i + 1 < mine) fetch(i + 1);
    float* tile = tiles + (size_t)(i % RING) * N * V;
    const float* row = rows + (i & 1) * row_len;
    const float d = row[2 * V], dec = row[2 * V + 1];
    float4 x = *(const float4*)(row + c4), y = make_float4(0.f, 0.f, 0.f, 0.f);
    x.x *= d; x.y *= d; x.z *= d; x.w *= d;
#pragma unroll 4
    for (int n = r0; n < N; n += rows_at_once) {
      float4 q = *(const float4*)(tile + n * V + c4);
      const float b = row[at_b + n], c = row[at_b + N + n];
      q.x = fmaf(dec, q.x, b * x.x); q.y = fmaf(dec, q.y, b * x.y); q.z = fmaf(dec, q.z, b * x.z); q.w = fmaf(dec, q.w, b * x.w);
      *(float4*)(tile + n * V + c4) = q;
      y.x = fmaf(c, q.x, y.x); y.y = fmaf(c, q.y, y.y); y.z = fmaf(c, q.z, y.z); y.w = fmaf(c, q.w, y.w);
    }
    for (int o = per; o < 32; o <<= 1) {                        // the rows that a warp's lanes share out
      y.x += __shfl_xor_sync(0xffffffffu, y.x, o);
      y.y += __shfl_xor_sync(0xffffffffu, y.y, o);
      y.z += __shfl_xor_sync(0xffffffffu, y.z, o);
      y.w += __shfl_xor_sync(0xffffffffu, y.w, o);
    }
    if (lane < per) *(float4*)(red + warp * V + c4) = y;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (!__syncthreads_and(ok)) {                               // the states are done, and the warps' sums are there, unless a wait ran out
      volatile int never = 0;
      if (tid == 0)
        for (int j = i; j < min(mine, i + RING - 1); j++) mbar_wait(full + 8 * (j % RING), (j / RING) & 1, &never);
      ok = false;
      break;
    }
    int b, h;
    pair(i, b, h);
    if (tid == 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(job.place(b, h)), "r"(smem_u32(tile)), "r"(tile_bytes) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      if (i + RING - 1 < mine) {                                // its place was pair i - 1's: read out by now, or waited for
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        load(i + RING - 1);
      }
    }
    if (tid < V) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; w++) s += red[w * V + tid];
      job.finish(b, h, tid, s, row[tid], row[V + tid]);
    }
    if (i + 1 < mine) stash(i + 1);
    __syncthreads();
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (!ok && err) atomicExch(err, 5);
}

// One row for each of n_seqs sequences. Two blocks an SM where their rings fit.
template <typename Job>
static int launch(const Job& job, int rows, int cols, int units, int sm_count, int* err, cudaStream_t stream) {
  const size_t smem = smem_bytes(rows, cols);
  cudaError_t e = smem <= SLLM_SMEM_UNASKED ? cudaSuccess : cudaFuncSetAttribute(state_step_kernel<Job>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
  if (e != cudaSuccess) return (int)e;
  const int most = (smem <= 112 * 1024 ? 2 : 1) * sm_count;
  state_step_kernel<Job><<<units < most ? units : most, 256, smem, stream>>>(job, units, err);
  SLLM_RETURN_LAST();
}

}  // namespace step
