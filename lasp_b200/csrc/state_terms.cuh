// States of the full-precision path as its output kernels take them: an fp32 number as the sum of three bf16 numbers
// (split_kernels.cu).  The scan that writes a state writes its terms: each is an operand of one or two products, and the
// arithmetic costs the scan, which memory bounds, nothing.
#pragma once
#include "common.cuh"

namespace lasp {

// The terms' sum is x, for infinities and NaN too; the first term of a finite x stays finite.
__device__ __forceinline__ void state_terms(float x, float (&t)[3]) {
  const float largest = __uint_as_float(0x7F7F0000u);   // of bf16
  const bool finite = isfinite(x);
  t[0] = __bfloat162float(__float2bfloat16_rn(finite ? fminf(fmaxf(x, -largest), largest) : x));
  float r = finite ? x - t[0] : 0.f;
  t[1] = __bfloat162float(__float2bfloat16_rn(r));
  r -= t[1];
  t[2] = r;   // (rounded where it is stored: what is left of 24 bits)
}
__device__ __forceinline__ float state_of_terms(const __nv_bfloat16* p, size_t i, size_t elems) {
  return (__bfloat162float(p[i + 2 * elems]) + __bfloat162float(p[i + elems])) + __bfloat162float(p[i]);
}
// four neighbouring elements of a state of `elems` elements, from element `el` on
__device__ __forceinline__ void store_state_terms(__nv_bfloat16* state, size_t el, size_t elems, float4 v) {
  float x[3], y[3], z[3], w[3];
  state_terms(v.x, x), state_terms(v.y, y), state_terms(v.z, z), state_terms(v.w, w);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x[i], y[i]), b = __floats2bfloat162_rn(z[i], w[i]);
    *reinterpret_cast<uint2*>(state + i * elems + el) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
}

}  // namespace lasp
