// Products of float matrices on the tcgen05 tensor cores, for kernels that make their operands on the chip.
//
// A float is the sum of three bfloat16 numbers, each the rounded rest of what the ones before it left: 8 + 8 + 8 bits of
// mantissa with signs of their own. A product of two such sums is taken as its six largest terms (0,0) (0,1) (1,0) (1,1) (0,2)
// (2,0), smallest first; what is left out, (1,2) and (2,1) above all, comes to 2^-24 of the product at most. Sums are float in tensor
// memory, where every step cuts what does not fit their 24 bits (FMA rounds it): of the largest term's up to eight steps of 128 deep
// that is some four halves of a last place, always towards zero. Against 64 bits, products of 128 deep this way / on the FMA units:
// linear attention's state 1.1e-7 / 1.2e-6 off (whose chain there is the longer one), the delta rule's outputs and state 2.1e-7 and
// 1.2e-7 / 9.7e-8 and 6.6e-8 (128 dims; of 32 dims 1.5e-7 and 1.1e-7 / 1.0e-7 and 7.9e-8; with decays near 1 2.8e-7 and 2.3e-7 /
// 2.0e-7 and 1.9e-7). Ending a sum half way and adding the halves as floats took the outputs to 1.7e-7, left the state where it was
// and cost a seventh of the kernels' time. Long sums do lose by it: 9.1e-6 against 1.6e-6 over 8,192 terms, so the products of
// weights (gemm_split_tcgen05.cu) end a sum after 64.
//
// A tile is 128 rows of 128 columns: three planes of 32 KB, a plane two blocks of 64 columns, a block 128 rows of 128 bytes with
// the 128-byte swizzle. The same bytes are an operand whose contraction runs along the columns (K-major) or along the rows
// (MN-major); which one is said by the descriptors of the product.
#pragma once
#include "tcgen05.cuh"

namespace sm3 {

constexpr int TILE = 128;
constexpr uint32_t BLOCK_BYTES = TILE * 128, PLANE_BYTES = 2 * BLOCK_BYTES, TILE_BYTES = 3 * PLANE_BYTES;

// eight columns from c (a multiple of 8) of row r into the tile's three planes
__device__ __forceinline__ void put8(uint8_t* tile, int r, int c, const float (&f)[8]) {
  uint4 q[3];
  split_pair(f[0], f[1], q[0].x, q[1].x, q[2].x);
  split_pair(f[2], f[3], q[0].y, q[1].y, q[2].y);
  split_pair(f[4], f[5], q[0].z, q[1].z, q[2].z);
  split_pair(f[6], f[7], q[0].w, q[1].w, q[2].w);
  uint8_t* at = tile + (c >> 6) * BLOCK_BYTES + r * 128 + (((((uint32_t)c >> 3) & 7) ^ (r & 7)) << 4);
#pragma unroll
  for (int p = 0; p < 3; p++) *(uint4*)(at + p * PLANE_BYTES) = q[p];
}

// operand descriptors for step k (16 deep) of a plane
__device__ __forceinline__ uint64_t desc_cols(uint32_t plane, int k) {        // contraction along the columns
  return umma_desc_sw128(plane + (k >> 2) * BLOCK_BYTES + (k & 3) * 32);
}
__device__ __forceinline__ uint64_t desc_rows(uint32_t plane, int k) {        // contraction along the rows
  return umma_desc_sw128_mn(plane + k * 2048, BLOCK_BYTES);
}
// 128 x 128 products; a or b "rows": its contraction runs along its tile's rows
__host__ __device__ constexpr uint32_t idesc(bool a_rows, bool b_rows) {
  return umma_idesc_bf16(128, 128) | (a_rows ? 1u << 15 : 0u) | (b_rows ? 1u << 16 : 0u);
}
// planes of the six terms' factors, smallest term first, two bits each
constexpr uint32_t TERM_A = 2u | 0u << 2 | 1u << 4 | 1u << 6 | 0u << 8 | 0u << 10, TERM_B = 0u | 2u << 2 | 1u << 4 | 0u << 6 | 1u << 8 | 0u << 10;
// D = A B, `steps` of 16 deep, both operands tiles in shared memory; a converged warp issues it through one lane (in a
// branch of one lane a product of 48 steps took some 85 clocks a step to issue, not the 64 it takes). The loops stay loops: these kernels run through their code once a block, so code is fetched, not found.
template <bool A_ROWS, bool B_ROWS>
__device__ __forceinline__ void product(uint32_t tmem_d, uint32_t a, uint32_t b, int steps) {
  constexpr uint32_t id = idesc(A_ROWS, B_ROWS);
  const bool one = elect_one();
#pragma unroll 1
  for (int t = 0; t < 6; t++) {
    const uint32_t pa = a + (TERM_A >> 2 * t & 3) * PLANE_BYTES, pb = b + (TERM_B >> 2 * t & 3) * PLANE_BYTES;
#pragma unroll 4
    for (int k = 0; k < steps; k++)
      if (one) umma_bf16(tmem_d, A_ROWS ? desc_rows(pa, k) : desc_cols(pa, k), B_ROWS ? desc_rows(pb, k) : desc_cols(pb, k), id, (t | k) ? 1u : 0u);
  }
}
// the same with A in tensor memory: three planes of 64 columns (two bfloat16 of K each)
template <bool B_ROWS>
__device__ __forceinline__ void product_ta(uint32_t tmem_d, uint32_t tmem_a, uint32_t b, int steps) {
  constexpr uint32_t id = idesc(false, B_ROWS);
  const bool one = elect_one();
#pragma unroll 1
  for (int t = 0; t < 6; t++) {
    const uint32_t pa = tmem_a + (TERM_A >> 2 * t & 3) * 64, pb = b + (TERM_B >> 2 * t & 3) * PLANE_BYTES;
#pragma unroll 4
    for (int k = 0; k < steps; k++)
      if (one)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "r"(pa + k * 8), "l"(B_ROWS ? desc_rows(pb, k) : desc_cols(pb, k)), "r"(id), "r"((t | k) ? 1u : 0u) : "memory");
  }
}

// What every block of these kernels has: all of tensor memory, one barrier for the products it waits for, a flag of waits given
// up. Products are issued by warp 0 between `ready()` (operands written by all threads are visible to the tensor cores) and
// `commit()`; `done()` lets every thread wait for them.
struct Unit {
  uint32_t tmem, bar, phase;
  volatile int* abort;
  bool ok;
  // `head`: 16 bytes of shared memory [barrier 8][tmem slot 4][abort 4]
  __device__ __forceinline__ void open(uint8_t* head) {
    bar = smem_u32(head);
    uint32_t* slot = (uint32_t*)(head + 8);
    abort = (volatile int*)(head + 12);
    phase = 0;
    ok = true;
    if (threadIdx.x == 0) {
      mbar_init(bar, 1);
      *abort = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(512) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem = *slot;
  }
  __device__ __forceinline__ void ready() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  __device__ __forceinline__ void commit() {    // by the warp that issued the products
    if (elect_one()) umma_commit(bar);
  }
  __device__ __forceinline__ void done() {      // a wait given up is remembered; the block walks on to its end and raises the flag
    if (!mbar_wait(bar, phase & 1, abort)) ok = false;
    phase++;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  __device__ __forceinline__ void close(int* err) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    if (!ok && err) atomicExch(err, 4);
  }
};

}  // namespace sm3
