// The tangent that caps an attention's scores, c tanh(s / c), for a run of scores side by side.
#pragma once
#include "common.cuh"

namespace {
__device__ __forceinline__ float rcp_approx(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// Lambert's continued fraction, cut after five levels, for |y| <= TANH_SMALL:
//     tanh y = y - y a (315 + 14 a) / (945 + 420 a + 15 a^2),   a = y^2,
// off by y^10 / 9.8e6 at most (1.1e-8 at 0.8), and no branch: a thread's scores run side by side, where the library's
// function, with its branch in each, holds every score up (220 cycles a score in the attention with mixed heads).  Where a warp
// has a larger one, masked ones included, it takes tanh_capped, which gives the smaller ones the same bits: the form that a score
// takes depends on that score alone.
constexpr float TANH_SMALL = 0.8f;
__device__ __forceinline__ float tanh_small(float y) {
  const float a = y * y;
  const float c = a * fmaf(a, 14.f, 315.f) * rcp_approx(fmaf(a, fmaf(a, 15.f, 420.f), 945.f));
  return fmaf(-y, c, y);
}
__device__ __forceinline__ float tanh_capped(float y) { return fabsf(y) <= TANH_SMALL ? tanh_small(y) : tanhf(y); }
}  // namespace
