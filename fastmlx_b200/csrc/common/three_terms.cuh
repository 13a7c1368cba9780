// A 32-bit value as the sum of three bfloat16 values (8 + 8 + 8 bits of its 24).
#pragma once
#include "common.cuh"

namespace {
// (x, y) -> three pairs of bfloat16 whose sums are x and y (to 2^-27 of them)
__device__ __forceinline__ void three_terms(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float2 hf = __bfloat1622float2(h);
  const float rx = x - hf.x, ry = y - hf.y;
  const __nv_bfloat162 m = __floats2bfloat162_rn(rx, ry);
  const float2 mf = __bfloat1622float2(m);
  const __nv_bfloat162 l = __floats2bfloat162_rn(rx - mf.x, ry - mf.y);
  hi = *reinterpret_cast<const unsigned*>(&h);
  mid = *reinterpret_cast<const unsigned*>(&m);
  lo = *reinterpret_cast<const unsigned*>(&l);
}

// The same for values of any size: an infinity is its own first term (and has no others: inf - inf would make a NaN of it), and a
// number that would round to one keeps the largest bfloat16 as its first term.
__device__ __noinline__ void three_terms_large(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
  unsigned t[2][3];
  const float v[2] = {x, y};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    bf16 h = __float2bfloat16_rn(v[i]);
    if (isinf(__bfloat162float(h)) && !isinf(v[i])) h = __ushort_as_bfloat16((unsigned short)(v[i] < 0.f ? 0xff7fu : 0x7f7fu));
    const float r = isinf(v[i]) ? 0.f : v[i] - __bfloat162float(h);
    const bf16 m = __float2bfloat16_rn(r), l = __float2bfloat16_rn(r - __bfloat162float(m));
    t[i][0] = __bfloat16_as_ushort(h); t[i][1] = __bfloat16_as_ushort(m); t[i][2] = __bfloat16_as_ushort(l);
  }
  hi = t[0][0] | t[1][0] << 16; mid = t[0][1] | t[1][1] << 16; lo = t[0][2] | t[1][2] << 16;
}
}  // namespace
