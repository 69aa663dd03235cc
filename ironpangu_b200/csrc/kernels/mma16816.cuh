// Warp-level pieces of the decode attention kernels and the greedy head: 16-byte asynchronous copies into shared memory, ldmatrix, the m16n8k16 bf16 product and weights as
// three bf16 terms. (Decode attention is bound by its keys' bytes; these products keep up with them at sixteen query rows.)
#pragma once
#include "common.cuh"

namespace ifab {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes, or zeros where `live` is false
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// one product alone
__device__ __forceinline__ void mma16816_alone(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ float two_sum(float& s, float b) {      // s += b; what the rounding leaves over (Knuth, The Art of Computer Programming 2, 4.2.2)
  const float a = s;
  s = a + b;
  const float c = s - a;
  return (a - (s - c)) + (b - c);
}
// Weights of a softmax as three bf16 terms each, which add up to all 24 bits of a weight. The first two are cut off below the value, not rounded to it, so that
// no term is 0 and none is negative: an infinite value of a key then stays infinite (inf * 0 is NaN, as is inf - inf). For that a weight is at least e^-62,
// from where on every term is a normal bf16 value; beside the weight of 1 that each softmax has, that is nothing, and so it serves for keys that are not there,
// too, whose values are read as zeros.
constexpr float LEAST_WEIGHT = 1.18e-27f;
__device__ __forceinline__ float weight_of(float x) {       // e^x; NaN stays NaN
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x) : "f"(-62.f));
  return __expf(x);
}
__device__ __forceinline__ float cut(float w) { return __uint_as_float((__float_as_uint(w) - 1u) & 0xffff0000u); }
__device__ __forceinline__ uint32_t upper_halves(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
// `last`: a power of two that the third term is multiplied by
__device__ __forceinline__ void three_terms(float a, float b, uint32_t (&t)[3], float last = 1.f) {
  const float a0 = cut(a), b0 = cut(b), ra = a - a0, rb = b - b0, a1 = cut(ra), b1 = cut(rb);
  t[0] = upper_halves(a0, b0);
  t[1] = upper_halves(a1, b1);
  t[2] = upper_halves((ra - a1) * last, (rb - b1) * last);
}

}  // namespace ifab
