// cnn_tc.cuh -- Blackwell tensor-core (tcgen05 / TMEM) building blocks for
// the warm-start network's implicit-GEMM convolutions.
//
// One CTA of 128 threads computes a 128 x N tile of D = A B^T (BF16 inputs,
// FP32 accumulator in tensor memory).  Operand tiles are staged in shared
// memory by the CTA's threads in the canonical no-swizzle ("interleaved")
// layouts the MMA descriptors describe, 64 K elements per stage, two stages:
// the threads gather stage s+1 while the tensor core works on stage s.  One
// elected thread issues tcgen05.mma and commits each stage to an mbarrier.
//
// Shared-memory operand layouts (element = 2 bytes, T = 8 elements = 16 B):
//   K-major  (row r of the M or N dimension, K index k):
//       byte (k/8) * (ROWS*16) + r*16 + (k%8)*2
//       descriptor: leading byte offset (between the two 8-element K halves of
//       one MMA) = ROWS*16, stride byte offset (between 8-row groups) = 128.
//   MN-major (row r, K index k):
//       byte (k/8) * (ROWS*16) + (r/8)*128 + (k%8)*16 + (r%8)*2
//       descriptor: leading byte offset (between 8-element K groups) = ROWS*16,
//       stride byte offset (between 8-row groups) = 128.
// In both, one MMA (K = 16) spans two 8-element K groups, so the descriptor
// start address advances by 2*ROWS*16 bytes per MMA along K.
// Descriptor bit layout and instruction-descriptor fields follow the sm100
// UMMA definitions (CUTLASS cute/arch/mma_sm100_desc.hpp).
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace xtc {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, no swizzle, sm100 version 1
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// instruction descriptor: BF16 x BF16 -> F32, M = 128, N, majors (0 = K, 1 = MN)
__host__ __device__ constexpr uint32_t idesc_bf16(int n, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
      :
      : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}

__device__ __forceinline__ void mma_commit(uint64_t *mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
               : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t *mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// bounded wait for the mbarrier phase with the given parity; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t *mbar, uint32_t parity, long long limit = 1ll << 26) {
  const uint32_t a = smem_u32(mbar);
  for (long long i = 0; i < limit; i++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The warp that issues MMAs runs as a whole and lets one elected lane issue: with
// its waits' outcomes and its warp number known to be the same in every lane,
// descriptors and counters stay in uniform registers, from which tcgen05.mma takes
// its operands.  Under `if (lane == 0)` an issue cost about 200 cycles, the same for
// N = 16 and 256: the halo convolution 32 -> 80 of 1048576 voxels took 573 us, 325
// with this.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(p));
  return p != 0;
}
// bounded wait of a whole warp
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *mbar, uint32_t parity, long long limit) {
  return __all_sync(0xffffffffu, mbar_wait(mbar, parity, limit));
}

// the single arrival of a transaction barrier, announcing `bytes` to come
__device__ __forceinline__ void mbar_expect_tx(uint64_t *mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// TMA tiled load of a 5-D box into shared memory, completing on mbar
__device__ __forceinline__ void tma_load_5d(void *dst, const void *tmap, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t *mbar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
      "%6}], [%7];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(mbar))
      : "memory");
}

// contiguous bulk copy global -> shared (16-byte aligned, size a multiple of 16)
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(mbar))
               : "memory");
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// TMEM allocation by one full warp; the base address lands in *dst (shared)
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
}

// 16 consecutive FP32 accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// zero 16 consecutive FP32 accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st16_zero(uint32_t taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1};" ::"r"(taddr),
      "r"(0u)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 16 BF16 values (or 8 FP32 values) to global memory: one 32-byte store, a whole
// sector, where p is 32-byte aligned; two 16-byte ones otherwise.  (An
// accumulator's lanes lie kilobytes apart: half sectors cost the tile kernel's
// forward pass at 512^2 x 64 0.6 of 8.9 ms.)
__device__ __forceinline__ void store32(void *p, const int4 &a, const int4 &b) {
  if ((reinterpret_cast<uintptr_t>(p) & 31) == 0) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                 "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
  } else {
    reinterpret_cast<int4 *>(p)[0] = a;
    reinterpret_cast<int4 *>(p)[1] = b;
  }
}

// TMEM columns to allocate for N accumulator columns (power of two, >= 32)
__host__ __device__ constexpr uint32_t tmem_cols(int n) {
  return n <= 32 ? 32u : n <= 64 ? 64u : n <= 128 ? 128u : 256u;
}

}  // namespace xtc
