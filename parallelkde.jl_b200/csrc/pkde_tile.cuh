// Shared-memory tiles by byte address: strided accesses then cost one 32-bit addition each.
#pragma once

#include "pkde_lines.cuh"

namespace pkde {

__device__ __forceinline__ unsigned smem_of(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ double2 lds(unsigned a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts(unsigned a, double2 v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned dst, const double2 *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// The radix-R combine's product: as the engine's, it fuses the other product of the imaginary part.
__device__ __forceinline__ double2 combine_cmul(double2 v, double2 w) {
  return make_double2(__fma_rn(v.x, w.x, -__dmul_rn(v.y, w.y)), __fma_rn(v.x, w.y, __dmul_rn(v.y, w.x)));
}

}  // namespace pkde
