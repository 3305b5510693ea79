// Warp-level matrix instructions, for attention over so few queries that a 128-row tcgen05 tile would be padding.
#pragma once

#include <type_traits>

#include "fm_common.cuh"

namespace fm {

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// Results of these depend on their operands alone (no volatile): the compiler may interleave independent ones, and the
// callers issue them so that a product does not wait for the one before it (about 35 cycles each).
// c[16 x 8] += a[16 x 16] b[16 x 8], 16-bit operands of type T, FP32 accumulation
template <typename T>
__device__ __forceinline__ void mma_16x8x16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __half>::value)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same over 32 values of K that lie together: lo and hi are a lane's eight (8 (lane % 4) .. of 32) of rows g and g + 8 of the first operand, b its
// eight of row g of the second, g = lane / 4.  K is permuted alike in both, which a sum does not mind.
template <typename T>
__device__ __forceinline__ void mma_16x8x32(float (&c)[4], const uint4& lo, const uint4& hi, const uint4& b) {
  const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
  mma_16x8x16<T>(c, a0, b.x, b.y);
  mma_16x8x16<T>(c, a1, b.z, b.w);
}
// Transpose of an 8 x 8 matrix of 16-bit values spread over the warp as fragments are (row lane / 4, columns 2 (lane % 4) ..).
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

}  // namespace fm
