// Shared by the fused W4A16 GEMMs: packed nibbles to fp16 operands, eight-column stores, ring cursors.
#pragma once

#include "common.cuh"

namespace xqt_b200 {

template <typename OutT>
__device__ __forceinline__ void w4f_store8(OutT* dst, const float (&v)[8]);
template <>
__device__ __forceinline__ void w4f_store8<__nv_bfloat16>(__nv_bfloat16* dst, const float (&v)[8]) {
  uint4 o;
  __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  __nv_bfloat162 c = __floats2bfloat162_rn(v[4], v[5]), d = __floats2bfloat162_rn(v[6], v[7]);
  o.x = *reinterpret_cast<uint32_t*>(&a); o.y = *reinterpret_cast<uint32_t*>(&b);
  o.z = *reinterpret_cast<uint32_t*>(&c); o.w = *reinterpret_cast<uint32_t*>(&d);
  *reinterpret_cast<uint4*>(dst) = o;
}
template <>
__device__ __forceinline__ void w4f_store8<__half>(__half* dst, const float (&v)[8]) {
  uint4 o;
  __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
  __half2 c = __floats2half2_rn(v[4], v[5]), d = __floats2half2_rn(v[6], v[7]);
  o.x = *reinterpret_cast<uint32_t*>(&a); o.y = *reinterpret_cast<uint32_t*>(&b);
  o.z = *reinterpret_cast<uint32_t*>(&c); o.w = *reinterpret_cast<uint32_t*>(&d);
  *reinterpret_cast<uint4*>(dst) = o;
}
template <typename T>
__device__ __forceinline__ void w4f_load8(const T* src, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(src);
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = to_float<T>(e[i]);
}

// 8 nibbles of `word` (k0..k7, canonical order) -> fp16 (code - zero) * scale as 4 registers in K order
__device__ __forceinline__ uint4 w4f_dequant_word(uint32_t word, __half2 off2, __half2 scale2) {
  uint32_t d[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;\n" : "=r"(r) : "r"(word >> (4 * i)), "n"(0x000f000f), "n"(0x64006400));
    __half2 v = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&r), off2), scale2);   // (k_i, k_{i+4})
    d[i] = *reinterpret_cast<uint32_t*>(&v);
  }
  uint4 o;
  o.x = __byte_perm(d[0], d[1], 0x5410);   // (k0, k1)
  o.y = __byte_perm(d[2], d[3], 0x5410);   // (k2, k3)
  o.z = __byte_perm(d[0], d[1], 0x7632);   // (k4, k5)
  o.w = __byte_perm(d[2], d[3], 0x7632);   // (k6, k7)
  return o;
}

// the same from a scale that fp16 does not hold: fp32 arithmetic, one rounding (`zero` includes the 1024 of the fast form)
static __device__ __noinline__ uint4 w4f_dequant_word_f32(uint32_t word, float zero, float scale) {
  uint32_t d[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 v = __floats2half2_rn(((float)((word >> (8 * i)) & 15u) + 1024.f - zero) * scale, ((float)((word >> (8 * i + 4)) & 15u) + 1024.f - zero) * scale);
    d[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
  return make_uint4(d[0], d[1], d[2], d[3]);
}

// Position in a ring of `n` slots that is walked in fixed steps: slot index and phase parity kept incrementally (a
// runtime `it % n` / `it / n` pair per stage is two integer divisions on every role's critical path).
struct W4FRing {
  uint32_t slot, phase, n;
  __device__ __forceinline__ W4FRing(uint32_t start, uint32_t slots) : slot(start % slots), phase((start / slots) & 1u), n(slots) {}
  __device__ __forceinline__ void advance(uint32_t step) {
    slot += step;
    while (slot >= n) { slot -= n; phase ^= 1u; }
  }
};

}  // namespace xqt_b200
