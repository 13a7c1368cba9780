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

// Warps of a block that bring the operands and do nothing else, and how far ahead.  One warp's 16-byte copies come in at 17 to 21 bytes a
// clock: with one, the walk waited for its operands whatever it did with them.  Two for 64 rows of state, of whose blocks several share
// an SM and its registers.
template <int D> constexpr int COPY_THREADS = D > 64 ? 128 : 64;
__device__ __forceinline__ void copy16(void* dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0));
}
template <int BYTES, int THREADS> __device__ __forceinline__ void copy_bytes(unsigned char* dst, const unsigned char* src, int thread) {
#pragma unroll 8
  for (int e = thread * 16; e < BYTES; e += THREADS * 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst + e)), "l"(src + e));
}

// What a warp of the four that own 16 columns of state does: a quarter of the state's rows lives in its registers, S^T as accumulator
// tiles of 16 columns by 8 rows, and turns into the left operand of S^T k and S^T q where it lies.  Those products' sums over
// the quarters meet in shared memory as 32-bit numbers (2 KB a warp, where the whole state as fragments would be 6 of 64 rows, 12 of 128,
// for each warp to read).
constexpr int RED = 4 * 32;                      // float4 that a warp puts down: four tiles of 8 tokens
constexpr int LEFT_WORDS = 3 * (RUN / 16) * 32 * 4;        // 32-bit words of a 16 x 32 matrix of the columns' values as left fragments

template <int D> struct RunWarp {
  static constexpr int NS = D / 32, KQ = D / 64, LD = D + 8;        // tiles of 8 rows, of 16 rows in a quarter; a row of k or q
  float S[NS][4];
  unsigned f[KQ][3][4];                          // S^T's terms as left fragments
  int lane, w, row, two;                         // a thread's columns of S: row, row + 8; within a tile of 8: two, two + 1

  __device__ __forceinline__ void load(const float* sp) {           // sp: this quarter of the first column's row of state
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      const float2 x = *reinterpret_cast<const float2*>(sp + (long long)row * D + j * 8 + two);
      const float2 y = *reinterpret_cast<const float2*>(sp + (long long)(row + 8) * D + j * 8 + two);
      S[j][0] = x.x; S[j][1] = x.y; S[j][2] = y.x; S[j][3] = y.y;
    }
  }
  __device__ __forceinline__ void store(float* sp) const {
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      *reinterpret_cast<float2*>(sp + (long long)row * D + j * 8 + two) = make_float2(S[j][0], S[j][1]);
      *reinterpret_cast<float2*>(sp + (long long)(row + 8) * D + j * 8 + two) = make_float2(S[j][2], S[j][3]);
    }
  }
  __device__ __forceinline__ void terms() {
#pragma unroll
    for (int k = 0; k < KQ; ++k) {
      three_terms(S[2 * k][0], S[2 * k][1], f[k][0][0], f[k][1][0], f[k][2][0]);
      three_terms(S[2 * k][2], S[2 * k][3], f[k][0][1], f[k][1][1], f[k][2][1]);
      three_terms(S[2 * k + 1][0], S[2 * k + 1][1], f[k][0][2], f[k][1][2], f[k][2][2]);
      three_terms(S[2 * k + 1][2], S[2 * k + 1][3], f[k][0][3], f[k][1][3], f[k][2][3]);
    }
  }
  // this quarter's share of S^T rows^T, rows [32][LD] in three terms: put down per 8 tokens
  __device__ __forceinline__ void against(const bf16* rows, float4* red) const {
    float c[4][4];
    unsigned b[4][3][2 * KQ];
    const bf16* p = rows + w * (D / 4);
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        unsigned x[4];
        if (KQ == 1) {                           // 16 rows of state: one access for two tiles of 8 tokens
          if (n & 1) continue;
          ldmatrix4(x, p + (t * RUN + n * 8 + (lane & 7) + (lane >> 4) * 8) * LD + (lane >> 3 & 1) * 8);
          b[n][t][0] = x[0]; b[n][t][1] = x[1]; b[n + 1][t][0] = x[2]; b[n + 1][t][1] = x[3];
        } else {
          ldmatrix4(x, p + (t * RUN + n * 8 + (lane & 7)) * LD + (lane >> 3) * 8);
#pragma unroll
          for (int i = 0; i < 2 * KQ; ++i) b[n][t][i] = x[i];
        }
      }
    products<KQ, 1>(c, f, b);
#pragma unroll
    for (int n = 0; n < 4; ++n) red[w * RED + n * 32 + lane] = make_float4(c[n][0], c[n][1], c[n][2], c[n][3]);
  }
  // the four quarters' sum for this warp's 8 tokens
  __device__ __forceinline__ void gather(float (&v)[4], const float4* red) const {
    float4 p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = red[i * RED + w * 32 + lane];
    v[0] = (p[0].x + p[1].x) + (p[2].x + p[3].x); v[1] = (p[0].y + p[1].y) + (p[2].y + p[3].y);
    v[2] = (p[0].z + p[1].z) + (p[2].z + p[3].z); v[3] = (p[0].w + p[1].w) + (p[2].w + p[3].w);
  }
  // this warp's 8 tokens of a 16 x 32 matrix of the columns' values, as three terms of left fragments that all four warps read
  __device__ __forceinline__ void share(unsigned* dst, const float (&v)[4]) const {
    unsigned t[3][2];
    three_terms(v[0], v[1], t[0][0], t[1][0], t[2][0]);
    three_terms(v[2], v[3], t[0][1], t[1][1], t[2][1]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint2*>(dst + ((i * 2 + (w >> 1)) * 32 + lane) * 4 + (w & 1) * 2) = make_uint2(t[i][0], t[i][1]);
  }
  __device__ __forceinline__ void shared(unsigned (&x)[2][3][4], const unsigned* src, int tiles) const {
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (k < tiles)
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const uint4 u = *reinterpret_cast<const uint4*>(src + ((t * 2 + k) * 32 + lane) * 4);
          x[k][t][0] = u.x; x[k][t][1] = u.y; x[k][t][2] = u.z; x[k][t][3] = u.w;
        }
  }
  // out = A x for this warp's 8 tokens, A [32][PT_LD] lower triangular in three terms, x as left fragments
  __device__ __forceinline__ void lower(float (&out)[4], const bf16* A, const unsigned* src) const {
    unsigned b[1][3][4], x[2][3][4];
    float c[1][4];
#pragma unroll
    for (int t = 0; t < 3; ++t) ldmatrix4(b[0][t], A + (t * RUN + w * 8 + (lane & 7)) * PT_LD + (lane >> 3) * 8);
    const int tiles = 1 + (w >> 1);
    shared(x, src, tiles);
    products<2, 2>(c, x, b, tiles);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = c[0][i];
  }
  // S <- decay S + x^T rows for this quarter, x as left fragments; decay(j): of the rows j * 8 + two and the next
  template <typename F> __device__ __forceinline__ void add(const bf16* rows, const unsigned* src, F decay) {
    unsigned x[2][3][4];
    shared(x, src, 2);
    constexpr int N = 2;                         // tiles of 8 rows at a time
#pragma unroll
    for (int j = 0; j < NS; j += N) {
      unsigned b[N][3][4];
      float d[N][4];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int t = 0; t < 3; ++t)
#pragma unroll
          for (int n = 0; n < N; n += 2) {
            unsigned r[4];
            ldmatrix4_trans(r, rows + (t * RUN + k * 16 + (lane & 15)) * LD + w * (D / 4) + (j + n + (lane >> 4)) * 8);
            b[n][t][2 * k] = r[0]; b[n][t][2 * k + 1] = r[1]; b[n + 1][t][2 * k] = r[2]; b[n + 1][t][2 * k + 1] = r[3];
          }
      products<2, 2>(d, x, b);
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const float2 e = decay(j + n);
        S[j + n][0] = fmaf(S[j + n][0], e.x, d[n][0]); S[j + n][1] = fmaf(S[j + n][1], e.y, d[n][1]);
        S[j + n][2] = fmaf(S[j + n][2], e.x, d[n][2]); S[j + n][3] = fmaf(S[j + n][3], e.y, d[n][3]);
      }
    }
  }
};
}  // namespace
