// mma.sync on bfloat16 and what feeds it: fragments from shared memory, and 32-bit values as three bfloat16 parts.
#pragma once
#include <cuda_bf16.h>

namespace cbis {

__device__ __forceinline__ void mma_16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool TRANS>
__device__ __forceinline__ void ldm4(unsigned (&r)[4], const void* smem) {
  const unsigned at = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&p);
}
// Two values' parts, packed; what is left of the values after a part goes on to the next.
__device__ __forceinline__ void cut3(float a, float b, unsigned (&part)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    part[i] = pack_bf16(a, b);
    a -= __uint_as_float(part[i] << 16);
    b -= __uint_as_float(part[i] & 0xffff0000u);
  }
}

}  // namespace cbis
