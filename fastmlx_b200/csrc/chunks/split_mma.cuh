// Products of 32-bit matrices on the tensor cores: every operand as three bfloat16 terms (8 + 8 + 8 bits of its 24),
// six of the nine products of terms, summed in 32-bit.  What is left out lies 2^-24 below a product.
#pragma once
#include "packed.cuh"
#include "three_terms.cuh"

namespace {
// Lets a kernel have `bytes` (always the same for one kernel) of dynamic shared memory: asked for once per thread and device.
template <auto KERNEL> inline cudaError_t raise_shared(size_t bytes) {
  static thread_local int raised = -1;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess || device == raised) return e;
  e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) raised = device;
  return e;
}

__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldmatrix4(unsigned (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ldmatrix2_trans(unsigned (&r)[2], const bf16* p) {        // lanes 0 to 15 name the rows
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(unsigned (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}

// A 16 x 8 tile of sums, kept apart by size of the terms: chains of dependent products that do not wait for one another.
// Products of the leading terms are added up in rounded 32-bit sums: the tensor cores' own sums cut off, and of
// these products that would be seen.
struct Sums {
  float big[4], middle[4], small[4];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 4; ++i) big[i] = middle[i] = small[i] = 0.f;
  }
  // += a (16 x 16, three terms) . b (16 x 8, three terms; the k-tile's two registers are b[term][j], b[term][j + 1])
  template <int NB> __device__ __forceinline__ void add(const unsigned (&a)[3][4], const unsigned (&b)[3][NB], int j) {
    float now[4] = {0.f, 0.f, 0.f, 0.f};
    mma16816(now, a[0], b[0][j], b[0][j + 1]);
    mma16816(middle, a[0], b[1][j], b[1][j + 1]);
    mma16816(small, a[1], b[1][j], b[1][j + 1]);
    mma16816(middle, a[1], b[0][j], b[0][j + 1]);
    mma16816(small, a[0], b[2][j], b[2][j + 1]);
    mma16816(small, a[2], b[0][j], b[0][j + 1]);
#pragma unroll
    for (int i = 0; i < 4; ++i) big[i] += now[i];
  }
  __device__ __forceinline__ float at(int i) const { return big[i] + (middle[i] + small[i]); }
};

// The six products of terms of `tiles` tiles of 16 of the contraction, for N right operands side by side: c[n] = a . b[n], both in three
// terms (tile k's registers of b: b[n][term][2 k], b[n][term][2 k + 1]).  The tensor cores cut their sums off instead of rounding them,
// and of the leading terms' products that would be seen: those of each tile are a sum of their own, added up rounded; the small terms'
// products are CHAINS sums.  A product that waits for the one before it takes 21 clocks, one that does not 8.2: hence the sums side
// by side, and the steps over all N at a time.
template <int KT, int CHAINS, int N, int NB>
__device__ __forceinline__ void products(float (&c)[N][4], const unsigned (&a)[KT][3][4], const unsigned (&b)[N][3][NB], int tiles = KT) {
  constexpr int TA[5] = {2, 0, 1, 1, 0}, TB[5] = {0, 2, 1, 0, 1};
  float big[KT][N][4], low[CHAINS][N][4];
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int k = 0; k < KT; ++k) big[k][n][i] = 0.f;
#pragma unroll
      for (int x = 0; x < CHAINS; ++x) low[x][n][i] = 0.f;
    }
#pragma unroll
  for (int s = 0; s < 5; ++s) {
#pragma unroll
    for (int k = 0; k < KT; ++k)
      if (k < tiles)
#pragma unroll
        for (int n = 0; n < N; ++n) mma16816(low[k % CHAINS][n], a[k][TA[s]], b[n][TB[s]][2 * k], b[n][TB[s]][2 * k + 1]);
    if (s < KT && s < tiles)
#pragma unroll
      for (int n = 0; n < N; ++n) mma16816(big[s % KT][n], a[s % KT][0], b[n][0][2 * (s % KT)], b[n][0][2 * (s % KT) + 1]);
  }
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float l = low[0][n][i], h = big[0][n][i];
#pragma unroll
      for (int x = 1; x < CHAINS; ++x) l += low[x][n][i];
#pragma unroll
      for (int k = 1; k < KT; ++k) h += big[k][n][i];
      c[n][i] = h + l;
    }
}
}  // namespace
