// Exact modular dot products on the tensor cores through byte limbs: shared helpers of the
// kernels that evaluate extension x base sums as u8 matrix products (k_sumcheck.cu,
// k_whir.cu). With x = sum_a 2^(8a) x_a and w = sum_b 2^(8b) w_b (bytes), sum_k w_k x_k =
// sum_(a,b) 2^(8(a+b)) sum_k w_(k,b) x_(k,a); each inner sum is accumulated in s32 by
// mma.m16n8k32 (at most 2^12 byte products per accumulator, below 2^28).
#pragma once
#include "common.cuh"
#include "poseidon2.cuh"

namespace wl {

#ifdef __CUDACC__
__device__ __forceinline__ void mma_u8_16832(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same as c = c0 + a b, free to move among other instructions.
__device__ __forceinline__ void mma_u8_16832_from(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int c0,
                                                  int c1, int c2, int c3) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}
// Byte a of four consecutive values, packed (limb a of a k-quad of the A fragment).
__device__ __forceinline__ void byte_transpose4(const uint4 q, uint32_t (&r)[4]) {
  const uint32_t p01l = __byte_perm(q.x, q.y, 0x5140), p01h = __byte_perm(q.x, q.y, 0x7362);
  const uint32_t p23l = __byte_perm(q.z, q.w, 0x5140), p23h = __byte_perm(q.z, q.w, 0x7362);
  r[0] = __byte_perm(p01l, p23l, 0x5410);
  r[1] = __byte_perm(p01l, p23l, 0x7632);
  r[2] = __byte_perm(p01h, p23h, 0x5410);
  r[3] = __byte_perm(p01h, p23h, 0x7632);
}

#endif

}  // namespace wl
