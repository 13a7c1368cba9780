// What the recurrences in runs of 32 tokens share: the layout of a run's 32 x 32 matrices, the solution of its triangular system,
// and the sums over earlier tokens where a value is not finite.
#pragma once
#include "split_mma.cuh"

namespace {
constexpr int RUN = 32;                         // tokens of a run
// Rows of the workspaces are as far apart as the kernels that walk the runs want them in shared memory (eight 16-byte pieces of
// eight rows meet no bank twice), so that a run's operands are runs of bytes to copy.
constexpr int PT_LD = RUN + 8;
constexpr int GRAM_LD = RUN + 4;
constexpr int PLANE = 3 * RUN * PT_LD;          // bf16 of one 32 x 32 matrix in three terms

// A warp turns M (strictly lower triangular, rows GRAM_LD apart) into T diag(beta), T = (1 + M)^-1: lane j solves for column j
// from the top down, T_ij = [i = j] - sum_{l < i} M_il T_lj, and its column takes beta_j.
__device__ __forceinline__ void solve_unit_lower(float* M, int lane, float beta) {
  float T[RUN];
#pragma unroll
  for (int i = 0; i < RUN; ++i) {
    float p[4] = {lane == i ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int l = 0; l < i; l += 4) {
      const float4 m = load4(M + i * GRAM_LD + l);
      p[0] = fmaf(-m.x, T[l], p[0]);
      if (l + 1 < i) p[1] = fmaf(-m.y, T[l + 1], p[1]);
      if (l + 2 < i) p[2] = fmaf(-m.z, T[l + 2], p[2]);
      if (l + 3 < i) p[3] = fmaf(-m.w, T[l + 3], p[3]);
    }
    T[i] = (p[0] + p[1]) + (p[2] + p[3]);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < RUN; ++i) M[i * GRAM_LD + lane] = T[i] * beta;
  if (__any_sync(0xffffffffu, !(beta - beta == 0.f))) {         // above the diagonal stays zero, whatever a later token's beta is
#pragma unroll 1
    for (int i = 0; i < lane; ++i) M[i * GRAM_LD + lane] = 0.f;
  }
  __syncwarp();
}

// Do the 128 threads of barrier `id` meet with `mine` true in any of them?
__device__ __forceinline__ bool meet_any(int id, bool mine) {
  int any;
  asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n barrier.cta.red.or.aligned.pred q, %2, 128, p;\n selp.s32 %0, 1, 0, q;\n}\n"
               : "=r"(any) : "r"((int)mine), "r"(id) : "memory");
  return any != 0;
}

__device__ __forceinline__ bool not_finite(const float (&v)[4]) {
  return !((v[0] - v[0]) + (v[1] - v[1]) + (v[2] - v[2]) + (v[3] - v[3]) == 0.f);
}

// out[i] = sum_{s <= t} A[t][s] x[s][col] for tokens t = t0 + (i & 1) and columns col = row + 8 (i >> 1), A lower triangular, x as left
// fragments of 16 columns by 32 tokens.  A product of matrices multiplies the zeros above the diagonal too, and zero times an
// infinity or a NaN of a later token would reach the tokens in front of it: runs that hold such a value take these sums instead.
__device__ __forceinline__ void lower_sums(float (&out)[4], const bf16* A, const unsigned* x, int t0, int row) {
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = 0.f;
#pragma unroll 1
  for (int s = 0; s <= t0 + 1; ++s) {
    float a[2] = {0.f, 0.f}, v[2] = {0.f, 0.f};
#pragma unroll
    for (int term = 2; term >= 0; --term)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[i] += __bfloat162float(A[(term * RUN + t0 + i) * PT_LD + s]);
        const unsigned* two = x + ((term * 2 + (s >> 4)) * 32 + row * 4 + ((s & 7) >> 1)) * 4 + (s >> 3 & 1) * 2 + i;
        v[i] += __bfloat162float(reinterpret_cast<const bf16*>(two)[s & 1]);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (s <= t0 || (i & 1)) out[i] = fmaf(a[i & 1], v[i >> 1], out[i]);
  }
}
}  // namespace
