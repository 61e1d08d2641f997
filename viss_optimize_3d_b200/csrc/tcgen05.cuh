// tcgen05.cuh -- the few fifth-generation tensor core operations this library
// uses: TF32 matrix products with FP32 accumulators in tensor memory.
//
// Operands lie in shared memory in the K-major layout without swizzle: core
// matrices of 8 rows x 16 bytes (4 TF32 values along K), 128 contiguous bytes;
// core matrices adjacent along the rows 128 bytes apart, along K `lbo` bytes.
#pragma once

#include "viss_common.cuh"

namespace viss {

// Byte offset of element (row, k).
__device__ __forceinline__ int umma_offset(int row, int k, int lbo) {
  return (k >> 2) * lbo + (row >> 3) * 128 + (row & 7) * 16 + (k & 3) * 4;
}

// Shared-memory matrix descriptor (no swizzle): start, stride along K, stride
// along the rows, in 16-byte units; bit 46 is the descriptor's fixed version bit.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, int lbo) {
  return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | (static_cast<uint64_t>((lbo >> 4) & 0x3fff) << 16) |
         (static_cast<uint64_t>(128 >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor: FP32 accumulator, TF32 operands, both K-major, M = 128.
__device__ __forceinline__ uint32_t umma_idesc_tf32(int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | ((128u >> 4) << 24);
}

// D (128 x n at tensor-memory address d) = or += A (128 x 8) B (n x 8)^T; one thread issues it.
__device__ __forceinline__ void umma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(static_cast<uint32_t>(add))
      : "memory");
}

// Arrives on `bar` when the thread's products issued so far are done.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

// Tensor memory of `cols` columns (a power of two >= 32); a whole warp calls
// both.  The address is written to shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
}

// Ordering around thread synchronisation, and of shared-memory writes before
// the tensor core (async proxy) reads them.
__device__ __forceinline__ void umma_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 (32) consecutive columns of the calling warp's 32 rows (warp w of the CTA
// reads rows 32 (w mod 4) ..): v[i] = row `lane`, column i.
__device__ __forceinline__ void tmem_load16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// x = hi + lo to 22 bits, each half a TF32 value (rounded to nearest).
__device__ __forceinline__ void split_tf32(float x, float &hi, float &lo) {
  uint32_t h, l;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
  hi = __uint_as_float(h);
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(x - hi));
  lo = __uint_as_float(l);
}

}  // namespace viss
