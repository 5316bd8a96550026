// f32 products on the tensor cores: operands in two tf32 parts, three MMAs per product.
#pragma once

#include "sm100.cuh"

namespace rt {
namespace {

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// ... and into zeros.
__device__ __forceinline__ void mma_tf32_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// x = hi + lo, both rounded to the 11 bits that the tensor core reads.  Only hi is rounded on the bit
// pattern: adding to the pattern carries a NaN of all ones (0x7fffffff, the one GPU arithmetic
// makes) past the exponent into a zero.  What is left has at most 12 bits, and times 1 + 2^-11 it is
// rounded once the bits past the eleventh are cut off; it is NaN for a NaN or an infinite x, so that
// a product with such an operand is NaN whatever became of hi.
__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  const float rest = x - __uint_as_float(hi);
  lo = __float_as_uint(fmaf(rest, 0x1p-11f, rest));
}

// 16 bytes to shared memory in the background; zeros if !read.
__device__ __forceinline__ void copy_async16(float* dst, const float* src, bool read) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sm100::smem_u32(dst)), "l"(src),
               "r"(read ? 16 : 0)
               : "memory");
}

}  // namespace
}  // namespace rt
