// Packed bf16 arithmetic shared by the kernels of the single-GPU layer, and the products of the decode kernels.
#pragma once

#include <cstdint>
#include <cuda_bf16.h>

#include <mscclpp/device/ptx.cuh>

namespace mscclpp {

// Packed bf16 arithmetic for the element-wise parts of the single-GPU layer. With a dozen warps per SM these loops are
// bound by instruction latency, not by memory: one HADD2 / HMUL2 / HFMA2 per two elements instead of a convert - operate -
// convert chain per element is what makes them fit in the shadow of the MMAs.
MSCCLPP_DEVICE_INLINE __nv_bfloat162 asBf162(uint32_t w) { return *reinterpret_cast<__nv_bfloat162*>(&w); }
MSCCLPP_DEVICE_INLINE uint32_t asWord(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
// a + b per element, each sum rounded once to bf16 (the adder works in fp32 internally: same result as an fp32 add + round)
MSCCLPP_DEVICE_INLINE uint4 addBf16x8(uint4 a, uint4 b) {
  return make_uint4(asWord(__hadd2(asBf162(a.x), asBf162(b.x))), asWord(__hadd2(asBf162(a.y), asBf162(b.y))),
                    asWord(__hadd2(asBf162(a.z), asBf162(b.z))), asWord(__hadd2(asBf162(a.w), asBf162(b.w))));
}
MSCCLPP_DEVICE_INLINE float sumSquaresBf16x8(uint4 v) {
  const float2 a = __bfloat1622float2(asBf162(v.x)), b = __bfloat1622float2(asBf162(v.y));
  const float2 c = __bfloat1622float2(asBf162(v.z)), d = __bfloat1622float2(asBf162(v.w));
  float s0 = a.x * a.x, s1 = b.x * b.x;
  s0 = fmaf(a.y, a.y, s0);
  s1 = fmaf(b.y, b.y, s1);
  s0 = fmaf(c.x, c.x, s0);
  s1 = fmaf(d.x, d.x, s1);
  s0 = fmaf(c.y, c.y, s0);
  s1 = fmaf(d.y, d.y, s1);
  return s0 + s1;
}
// v * g * s with the fp32 scale s split into a bf16 head and a bf16 tail (s = hi + lo up to 2^-17 relative), so that the
// result carries the two product roundings of bf16 arithmetic but not a third from rounding s itself.
MSCCLPP_DEVICE_INLINE uint32_t scaleBf16x2(uint32_t v, uint32_t g, __nv_bfloat162 hi, __nv_bfloat162 lo, bool hasGamma) {
  const __nv_bfloat162 p = hasGamma ? __hmul2(asBf162(v), asBf162(g)) : asBf162(v);
  return asWord(__hfma2(p, lo, __hmul2(p, hi)));
}

// Two fp32 values per instruction.
MSCCLPP_DEVICE_INLINE uint64_t pairOf(uint32_t bf16x2) {
  uint64_t p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "r"(bf16x2 << 16), "r"(bf16x2 & 0xffff0000u));
  return p;
}
MSCCLPP_DEVICE_INLINE uint64_t pairOf(float a, float b) {
  uint64_t p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a), "f"(b));
  return p;
}
MSCCLPP_DEVICE_INLINE float2 valuesOf(uint64_t p) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
MSCCLPP_DEVICE_INLINE uint64_t mulPair(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
MSCCLPP_DEVICE_INLINE uint64_t fmaPair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// ... rounded to bf16
MSCCLPP_DEVICE_INLINE uint32_t packPair(uint64_t p) {
  const float2 f = valuesOf(p);
  return asWord(__floats2bfloat162_rn(f.x, f.y));
}

// Warp-level tensor-core products of the decode kernels: four 8 x 8 matrices out of shared memory, and
// D[16 x 8] += A[16 x 16] (row-major) * B[16 x 8] (column-major), bf16 operands, fp32 accumulation.
MSCCLPP_DEVICE_INLINE void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
MSCCLPP_DEVICE_INLINE void mma_m16n8k16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

}  // namespace mscclpp
