// Linear recurrences with a matrix of 32-bit state per head, over portions, in runs of 32 tokens as matrix products.
//
//     S <- a_t S + k_t u_t^T;   o_t = S^T q_t;   u_t = v_t (weighed by a number per token), or the delta rule's
//     u_t = beta_t (v_t - (a_t S)^T k_t)
//
// with one decay a_t per head.  Within a run that starts from S, with A_t = a_1 ... a_t,
//
//     o_t = A_t S^T q_t + sum_{s <= t} (q_t . k_s) (A_t / A_s) u_s
//     u   = T diag(beta) (v - A (k S)),   T = (1 + strictly lower part of beta_t (k_t . k_s) (A_t / A_s))^-1
//     S  <- A_32 S + sum_s (A_32 / A_s) k_s u_s^T
//
// Ratios A_t / A_s are running products of decays (at most one, no logarithm, no division).  Every product that meets the
// state runs on the tensor cores with three bfloat16 terms an operand (split_mma.cuh), so that its errors are those of the walk
// token by token in 32-bit multiply-adds (the kernels of delta_rule.cu and ssm.cu; 2,048 tokens of the delta rule against 64-bit, of
// the result's norm: decays of 0.9 to 1 1.3e-7 either way, of 0.8 to 1 1.2e-7 here and 1.1e-7 there; plain write 1.1e-7 and 1.3e-7).
// That walk is one chain of dependent steps of some 250 ns a token; a run of 32 tokens here takes 1.4 us at 64 rows of state, 3.3 us at 128.  2,048
// tokens, 32 heads on 8 key heads, both kernels, walk and runs in us: one request of 64 x 64 delta rule 522 and 116, plain write 346 and
// 85; two of 128 x 128 937 and 227, 646 and 174; 64 heads of 64 values over 128 rows, one request 828 and 178, 1,777 tokens of five 560 and 171.
//
//   chunk_prepare  per (run, key group): k and q as three terms; k . k^T and q . k^T in 32-bit, and per head of the group
//                  the decayed q . k^T and T, as three terms.  All runs at once.
//   chunk_delta, chunk_plain   per (request, head, 16 or 32 columns of S): the runs in order.
//
// An infinity or a NaN reaches what the walk lets it reach, its own token and the ones behind it (in its own column where a value holds
// it), as a NaN: its second term is inf - inf.  A run that holds one sums over earlier tokens without the zeros of later ones (lower_sums).
#include <math.h>
#include "runs.cuh"

namespace {
// A run's operands: k and q of a group, and P, T and numbers of a head.
template <int D> constexpr int QK_LD = D + 8;
template <int D> constexpr int QK_SIZE = 2 * 3 * RUN * QK_LD<D>;              // bf16 of q and k of a run and group
template <bool DELTA> constexpr int PT_SIZE = (DELTA ? 2 : 1) * PLANE + 4 * RUN;   // P, T and, as floats, A_t and E_s

// The place of a row's first run in the workspaces: rows do not overlap, whatever their lengths.
__device__ __forceinline__ int first_run(int row_start, int r) { return row_start / RUN + r; }

// x [T, C]: q of group g at qoff + g D, k at koff + g D.  decay, weight: per token and head, rows of gstride.
// qk [run][G][q, k][3][32][D], pt [run][H][P, T (delta rule)][3][32][32] and floats [A_t: 32, E_s: 32].
// Warps of a block: a block of 128 rows fills a third of an SM's shared memory, and with eight warps its phases are half as long
// (1,777 tokens, 8 groups of 8 heads: 38 -> 31 us); of 64 rows five blocks of four warps share an SM (34 and 34 us).
template <int D> constexpr int PREP_WARPS = D > 64 ? 8 : 4;
template <int D, bool DELTA>
__global__ void __launch_bounds__(32 * PREP_WARPS<D>, D > 64 ? 2 : 5)          // as many blocks as shared memory holds
chunk_prepare_kernel(const float* x, long long C, int qoff, int koff, const float* decay, const float* weight, int gstride,
                     const int* row_start, int min_tokens, int H, int G, bf16* qk, bf16* pt, int lo, int hi) {
  constexpr int LD = D + 4, THREADS = 32 * PREP_WARPS<D>;
  extern __shared__ __align__(16) float psm[];
  float* qs = psm;                              // [32][LD]
  float* ks = qs + RUN * LD;
  float* qkm = ks + RUN * LD;                   // q . k^T, [32][GRAM_LD]
  float* kkm = qkm + RUN * GRAM_LD;             // k . k^T
  const int c = blockIdx.x, g = blockIdx.y, r = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* mine = kkm + RUN * GRAM_LD + warp * RUN * GRAM_LD;      // a warp's matrix
  pdl_wait();      // no early trigger: blocks of the walk would sit on the shared memory that this kernel's blocks want
  const int first = row_start[r], n = row_start[r + 1] - first;
  if (c * RUN >= n || n < min_tokens) return;
  const int t0 = first + c * RUN, cnt = min(RUN, n - c * RUN);
  const long long run = first_run(first, r) + c - lo;
  if (run < 0 || run >= hi - lo) return;         // a run of another wave
  bf16* planes = qk + (run * G + g) * QK_SIZE<D>;
  for (int e = tid; e < 2 * RUN * (D / 4); e += THREADS) {
    const int which = e / (RUN * (D / 4)), row = e / (D / 4) % RUN, d = e % (D / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < cnt) v = load4(x + (long long)(t0 + row) * C + (which ? koff : qoff) + g * D + d);
    store4((which ? ks : qs) + row * LD + d, v);
    unsigned a[3], b[3];
    three_terms(v.x, v.y, a[0], a[1], a[2]);
    three_terms(v.z, v.w, b[0], b[1], b[2]);
#pragma unroll
    for (int term = 0; term < 3; ++term)
      *reinterpret_cast<uint2*>(planes + ((which * 3 + term) * RUN + row) * QK_LD<D> + d) = make_uint2(a[term], b[term]);
  }
  __syncthreads();
  {
    constexpr int PER = THREADS / RUN, NC = RUN / PER;       // a thread's columns: s0, s0 + PER, ...; neighbours read neighbouring rows
    const int t = tid / PER, s0 = tid % PER;
    float tq[NC], tk[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) tq[j] = tk[j] = 0.f;
    auto fma4 = [](float4& c, float4 u, float4 v) {
      c.x = fmaf(u.x, v.x, c.x); c.y = fmaf(u.y, v.y, c.y); c.z = fmaf(u.z, v.z, c.z); c.w = fmaf(u.w, v.w, c.w);
    };
#pragma unroll 1
    for (int d0 = 0; d0 < D; d0 += 16) {        // sums of 16 products in four chains, then of those: as short chains as the walk's
      float4 aq[NC], ak[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) aq[j] = ak[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int d = d0; d < d0 + 16; d += 4) {
        const float4 q4 = load4(qs + t * LD + d), k4 = load4(ks + t * LD + d);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const float4 s4 = load4(ks + (s0 + PER * j) * LD + d);
          fma4(aq[j], q4, s4);
          if (DELTA) fma4(ak[j], k4, s4);
        }
      }
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        tq[j] += (aq[j].x + aq[j].y) + (aq[j].z + aq[j].w);
        if (DELTA) tk[j] += (ak[j].x + ak[j].y) + (ak[j].z + ak[j].w);
      }
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      qkm[t * GRAM_LD + s0 + PER * j] = tq[j];
      if (DELTA) kkm[t * GRAM_LD + s0 + PER * j] = tk[j];
    }
  }
  __syncthreads();
  auto emit = [&](bf16* dst) {                  // a warp's 32 x 32 matrix as three terms
#pragma unroll 2
    for (int row = lane >> 3; row < RUN; row += 4) {
      const int s = (lane & 7) * 4;
      const float4 v = load4(mine + row * GRAM_LD + s);
      unsigned a[3], b[3];
      three_terms(v.x, v.y, a[0], a[1], a[2]);
      three_terms(v.z, v.w, b[0], b[1], b[2]);
#pragma unroll
      for (int term = 0; term < 3; ++term)
        *reinterpret_cast<uint2*>(dst + (term * RUN + row) * PT_LD + s) = make_uint2(a[term], b[term]);
    }
  };
  const int per = H / G;
  for (int hh = warp; hh < per; hh += PREP_WARPS<D>) {
    const int h = g * per + hh;
    const bool live = lane < cnt;
    const float a = live ? decay[(long long)(t0 + lane) * gstride + h] : 1.f;
    const float w = live ? weight[(long long)(t0 + lane) * gstride + h] : 0.f;
    bf16* out = pt + (run * H + h) * PT_SIZE<DELTA>;
    float* sc = reinterpret_cast<float*>(out + (DELTA ? 2 : 1) * PLANE);
    float ratio = 0.f, cum = 1.f, own = 1.f;    // lane s: A_t / A_s as t goes on; A_t; A_lane
    float rows[RUN];
#pragma unroll
    for (int t = 0; t < RUN; ++t) {
      const float at = __shfl_sync(0xffffffffu, a, t), wt = __shfl_sync(0xffffffffu, w, t);
      cum *= at;
      if (lane == t) own = cum;
      ratio = lane < t ? ratio * at : lane == t ? 1.f : 0.f;
      // the decayed q . k^T, the weights of a plain write folded in
      mine[t * GRAM_LD + lane] = lane <= t ? qkm[t * GRAM_LD + lane] * ratio * (DELTA ? 1.f : w) : 0.f;
      if (DELTA) rows[t] = lane < t ? wt * kkm[t * GRAM_LD + lane] * ratio : 0.f;
    }
    sc[lane] = own;
    sc[RUN + lane] = DELTA ? ratio : ratio * w;
    __syncwarp();
    emit(out);
    __syncwarp();
    if (DELTA) {
#pragma unroll
      for (int t = 0; t < RUN; ++t) mine[t * GRAM_LD + lane] = rows[t];
      __syncwarp();
      solve_unit_lower(mine, lane, w);
      emit(out + PLANE);
      __syncwarp();
    }
  }
}

// Shared memory of chunk_delta: two stages of a run's operands, and what the four warps of 16 columns hand one another.
template <int D, int MT> struct DeltaSmem {
  static constexpr int V_LD = 16 * MT + 4;                                // floats
  static constexpr size_t STAGE = (size_t)(QK_SIZE<D> + PT_SIZE<true>) * 2 + (size_t)RUN * V_LD * 4;
  static constexpr int S_WORDS = 3 * (D / 16) * 32 * 4;                   // 32-bit words of S^T's fragments, per 16 columns
  static constexpr int U_WORDS = 3 * (RUN / 16) * 32 * 4;                 // of R's, U's and E's
  static constexpr size_t BYTES = 2 * STAGE + (size_t)MT * (S_WORDS + 3 * U_WORDS) * 4;
};

// grid (columns / (16 MT), H, R), 128 MT + 32 threads: four warps per 16 columns, and one that copies.  S^T is kept as
// accumulator tiles of 16 columns by 8 rows of state, a quarter of the rows in each warp; a warp works out the run's
// read-outs for 8 of its 32 tokens.  A product's left operand is always S^T or a 16 x 32 matrix of the columns' values:
// accumulators turn into the next product's left operand where they lie, and cross to the other warps through shared
// memory as finished fragments.  Bound by the latency of that chain (four exchanges a run), not by a unit: hence 32 tokens
// a run (64 take 1.2 times the products and 1.3 times the operands' bytes per token), four warps to share a link's
// products, and copies that no link waits for.
template <int D, int MT>
__global__ void __launch_bounds__(128 * MT + 32)
chunk_delta_kernel(const bf16* qk, const bf16* pt, const float* x, long long C, int voff, const int* row_start,
                  const int* row_slot, float* state, long long slot_stride, float* out, int min_tokens, int H, int G, int P, int max_slots,
                  int lo, int hi) {
  using Z = DeltaSmem<D, MT>;
  constexpr int KT = D / 16, NS = D / 32;        // k-tiles of S; 8-row tiles of S^T per warp
  extern __shared__ __align__(16) unsigned char csm[];
  const int r = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * 16 * MT;
  const int tid = threadIdx.x, lane = tid & 31, mt = tid >> 7, w = tid >> 5 & 3;
  pdl_wait();
  pdl_trigger();
  const int slot = row_slot[r];
  if (slot < 0 || slot >= max_slots) return;
  const int first = row_start[r], n = row_start[r + 1] - first;
  if (n < min_tokens) return;                    // walked token by token in a launch of its own
  const int place = first_run(first, r), g = h / (H / G);
  const int c_lo = max(0, lo - place), c_hi = min((n + RUN - 1) / RUN, hi - place);        // the row's runs of this wave
  if (c_lo >= c_hi) return;
  const long long run0 = place - lo;             // (of the row's first run, which may lie in front of the workspace)
  if (tid >= 128 * MT) {                         // the copying warp: a run's operands land while the run before it is walked
    auto cp16 = [](void* dst, const void* src, bool there) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0));
    };
    for (int c = c_lo; c < c_hi; ++c) {
      unsigned char* dst = csm + (c & 1) * Z::STAGE;
      const unsigned char* src = reinterpret_cast<const unsigned char*>(qk + ((run0 + c) * G + g) * QK_SIZE<D>);
#pragma unroll 8
      for (int e = lane * 16; e < QK_SIZE<D> * 2; e += 512) cp16(dst + e, src + e, true);
      dst += QK_SIZE<D> * 2;
      src = reinterpret_cast<const unsigned char*>(pt + ((run0 + c) * H + h) * PT_SIZE<true>);
#pragma unroll 8
      for (int e = lane * 16; e < PT_SIZE<true> * 2; e += 512) cp16(dst + e, src + e, true);
      float* dv = reinterpret_cast<float*>(dst + PT_SIZE<true> * 2);
#pragma unroll
      for (int e = lane; e < RUN * 4 * MT; e += 32) {
        const int t = e / (4 * MT), q = e % (4 * MT) * 4;
        const bool there = c * RUN + t < n;
        cp16(dv + t * Z::V_LD + q, x + (long long)(first + (there ? c * RUN + t : 0)) * C + voff + (long long)h * P + c0 + q, there);
      }
      asm volatile("cp.async.commit_group;\n" ::);
      asm volatile("cp.async.wait_group 0;\n" ::);
      __syncthreads();                           // run c is there; run c - 1 has been walked, and its stage is free
    }
    return;
  }
  unsigned* sfr = reinterpret_cast<unsigned*>(csm + 2 * Z::STAGE) + mt * Z::S_WORDS;
  unsigned* ufr = reinterpret_cast<unsigned*>(csm + 2 * Z::STAGE) + MT * Z::S_WORDS + mt * 3 * Z::U_WORDS;
  unsigned* efr = ufr + Z::U_WORDS;
  unsigned* rfr = efr + Z::U_WORDS;
  const int row = lane >> 2, two = (lane & 3) * 2;            // a thread's columns of S: row, row + 8; within a tile of 8: two, two + 1
  float* sp = state + (long long)slot * slot_stride + ((long long)h * P + c0 + mt * 16) * D + w * (D / 4);
  float S[NS][4];
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const float2 a = *reinterpret_cast<const float2*>(sp + (long long)row * D + j * 8 + two);
    const float2 b = *reinterpret_cast<const float2*>(sp + (long long)(row + 8) * D + j * 8 + two);
    S[j][0] = a.x; S[j][1] = a.y; S[j][2] = b.x; S[j][3] = b.y;
  }
  auto share_state = [&]() {                     // this warp's rows of state as left fragments, three terms
#pragma unroll
    for (int j = 0; j < NS; j += 2) {
      unsigned f[3][4];
      three_terms(S[j][0], S[j][1], f[0][0], f[1][0], f[2][0]);
      three_terms(S[j][2], S[j][3], f[0][1], f[1][1], f[2][1]);
      three_terms(S[j + 1][0], S[j + 1][1], f[0][2], f[1][2], f[2][2]);
      three_terms(S[j + 1][2], S[j + 1][3], f[0][3], f[1][3], f[2][3]);
#pragma unroll
      for (int t = 0; t < 3; ++t)
        *reinterpret_cast<uint4*>(sfr + ((t * KT + w * (NS / 2) + j / 2) * 32 + lane) * 4) = make_uint4(f[t][0], f[t][1], f[t][2], f[t][3]);
    }
  };
  auto share_tile = [&](unsigned* dst, const float (&v)[4]) {  // this warp's 8 tokens of a 16 x 32 matrix, likewise
    unsigned f[3][2];
    three_terms(v[0], v[1], f[0][0], f[1][0], f[2][0]);
    three_terms(v[2], v[3], f[0][1], f[1][1], f[2][1]);
#pragma unroll
    for (int t = 0; t < 3; ++t)
      *reinterpret_cast<uint2*>(dst + ((t * 2 + (w >> 1)) * 32 + lane) * 4 + (w & 1) * 2) = make_uint2(f[t][0], f[t][1]);
  };
  auto fragment = [&](unsigned (&f)[3][4], const unsigned* src, int tiles, int k) {
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const uint4 u = *reinterpret_cast<const uint4*>(src + ((t * tiles + k) * 32 + lane) * 4);
      f[t][0] = u.x; f[t][1] = u.y; f[t][2] = u.z; f[t][3] = u.w;
    }
  };
  share_state();
  const long long ostride = (long long)H * P;
  float* op = out + (long long)first * ostride + (long long)h * P + c0 + mt * 16;
  const int t0 = w * 8 + two;                    // this thread's tokens of a run: t0, t0 + 1
  const int rows8 = w * 8 + (lane & 7), quarter = (lane >> 3) * 8;
  for (int c = c_lo; c < c_hi; ++c) {
    __syncthreads();                             // the run's operands and S's fragments are there
    const bf16* dq = reinterpret_cast<const bf16*>(csm + (c & 1) * Z::STAGE);
    const bf16* dk = dq + 3 * RUN * QK_LD<D>;
    const bf16* dp = dq + QK_SIZE<D>;
    const float* ds = reinterpret_cast<const float*>(dp + 2 * PLANE);
    const float* dv = ds + 2 * RUN + mt * 16;
    const float A0 = ds[t0], A1 = ds[t0 + 1], E0 = ds[RUN + t0], E1 = ds[RUN + t0 + 1], last = ds[RUN - 1];
    float v[4] = {dv[t0 * Z::V_LD + row], dv[(t0 + 1) * Z::V_LD + row], dv[t0 * Z::V_LD + row + 8], dv[(t0 + 1) * Z::V_LD + row + 8]};
    // what the state in front of the run gives these 8 tokens: S^T q, and S^T k for the delta rule; side by side, so that one's
    // chains of products fill the other's waits
    Sums o, kS;
    o.zero();
    kS.zero();
    {
#pragma unroll
      for (int k2 = 0; k2 < KT / 2; ++k2) {
        unsigned bq[3][4], bk[3][4];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          ldmatrix4(bk[t], dk + (t * RUN + rows8) * QK_LD<D> + k2 * 32 + quarter);
          ldmatrix4(bq[t], dq + (t * RUN + rows8) * QK_LD<D> + k2 * 32 + quarter);
        }
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          unsigned a[3][4];
          fragment(a, sfr, KT, k2 * 2 + kk);
          kS.add(a, bk, kk * 2);
          o.add(a, bq, kk * 2);
        }
      }
    }
    {                                             // u = T diag(beta) (v - A (S^T k))
      unsigned bt[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t) ldmatrix4(bt[t], dp + PLANE + (t * RUN + rows8) * PT_LD + quarter);
      v[0] = fmaf(-A0, kS.at(0), v[0]); v[1] = fmaf(-A1, kS.at(1), v[1]);
      v[2] = fmaf(-A0, kS.at(2), v[2]); v[3] = fmaf(-A1, kS.at(3), v[3]);
      share_tile(rfr, v);
      const bool odd = meet_any(1 + mt, not_finite(v));
      Sums u;
      u.zero();
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (k <= (w >> 1)) {                      // T is lower triangular
          unsigned a[3][4];
          fragment(a, rfr, 2, k);
          u.add(a, bt, k * 2);
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = u.at(i);
      if (odd) lower_sums(v, dp + PLANE, rfr, t0, row);
    }
    const bool mine = not_finite(v);
    share_tile(ufr, v);
    v[0] *= E0; v[1] *= E1; v[2] *= E0; v[3] *= E1;
    share_tile(efr, v);
    const bool odd = meet_any(1 + mt, mine);
    // S <- A_32 S + sum_s (E_s u_s) k_s^T for this warp's rows of state, and what the run's own tokens give: the decayed
    // q . k^T times u
    Sums y, d[NS];
    y.zero();
    {
      unsigned bp[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t) ldmatrix4(bp[t], dp + (t * RUN + rows8) * PT_LD + quarter);
#pragma unroll
      for (int j = 0; j < NS; ++j) d[j].zero();
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        unsigned e[3][4], a[3][4];
        fragment(e, efr, 2, k);
        fragment(a, ufr, 2, k);
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          unsigned b[3][2];
#pragma unroll
          for (int t = 0; t < 3; ++t)
            ldmatrix2_trans(b[t], dk + (t * RUN + k * 16 + (lane & 15)) * QK_LD<D> + w * (D / 4) + j * 8);
          d[j].add(e, b, 0);
        }
        if (k <= (w >> 1)) y.add(a, bp, k * 2);
      }
    }
#pragma unroll
    for (int j = 0; j < NS; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) S[j][i] = fmaf(S[j][i], last, d[j].at(i));
    share_state();                                // the others' reads of these fragments lie in front of the last meeting
    const int t = c * RUN + t0;
    float res[4] = {y.at(0), y.at(1), y.at(2), y.at(3)};
    if (odd) lower_sums(res, dp, ufr, t0, row);
#pragma unroll
    for (int i = 0; i < 4; ++i) res[i] = fmaf(i & 1 ? A1 : A0, o.at(i), res[i]);
    if (t < n) {
      op[(long long)t * ostride + row] = res[0];
      op[(long long)t * ostride + row + 8] = res[2];
    }
    if (t + 1 < n) {
      op[(long long)(t + 1) * ostride + row] = res[1];
      op[(long long)(t + 1) * ostride + row + 8] = res[3];
    }
  }
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    *reinterpret_cast<float2*>(sp + (long long)row * D + j * 8 + two) = make_float2(S[j][0], S[j][1]);
    *reinterpret_cast<float2*>(sp + (long long)(row + 8) * D + j * 8 + two) = make_float2(S[j][2], S[j][3]);
  }
}

// Shared memory of chunk_plain: stages of a run's operands, and what the four warps of 16 columns hand one another: their shares of S^T q,
// and U and E as fragments.
template <int D, int MT> struct PlainSmem {
  static constexpr int V_LD = 16 * MT + 4;                                // floats
  static constexpr size_t STAGE = (size_t)(QK_SIZE<D> + PT_SIZE<false>) * 2 + (size_t)RUN * V_LD * 4;
  static constexpr int MEET = 4 * RED * 4 + 2 * LEFT_WORDS;               // 32-bit words per 16 columns
  static constexpr size_t bytes(int stages) { return stages * STAGE + (size_t)MT * MEET * 4; }
};

// The same without the delta rule, whose u is at hand before the run: nothing on the state's own chain crosses warps, so each warp keeps its
// quarter of the state's rows to itself (RunWarp).  Four warps copy (two for 64 rows), two stages of operands or three.  Bound by no unit: the tensor pipe is
// busy for 35 % of the time (1,777 tokens of five requests, 64 heads of 64 values over 128 rows; 105 products a warp and run, one every 8.2
// clocks of a scheduler where none waits for another, 21 where one does), and warps wait in turns for results of fixed latency, at the block's
// barriers, for that pipe and for operands.  With the state shared as fragments and one copying
// warp, which everything waited for: 1,777 tokens of five requests, 64 heads of 64 values over 128 rows 153 us, 138 here; 1,531 tokens of a
// retention with 32 heads of 64 x 64 77 and 51.  For the delta rule the meeting of the quarters stands on the chain: 92 us that way, 95 this.
template <int D, int MT>
__global__ void __launch_bounds__(128 * MT + COPY_THREADS<D>)
chunk_plain_kernel(const bf16* qk, const bf16* pt, const float* x, long long C, int voff, const float* skip, const int* row_start,
                  const int* row_slot, float* state, long long slot_stride, float* out, int min_tokens, int H, int G, int P, int max_slots,
                  int lo, int hi, int stages) {
  using Z = PlainSmem<D, MT>;
  extern __shared__ __align__(16) unsigned char csm[];
  const int r = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * 16 * MT;
  const int tid = threadIdx.x, lane = tid & 31, mt = tid >> 7, w = tid >> 5 & 3;
  pdl_wait();
  pdl_trigger();
  const int slot = row_slot[r];
  if (slot < 0 || slot >= max_slots) return;
  const int first = row_start[r], n = row_start[r + 1] - first;
  if (n < min_tokens) return;                    // walked token by token in a launch of its own
  const int place = first_run(first, r), g = h / (H / G);
  const int c_lo = max(0, lo - place), c_hi = min((n + RUN - 1) / RUN, hi - place);        // the row's runs of this wave
  if (c_lo >= c_hi) return;
  const long long run0 = place - lo;             // (of the row's first run, which may lie in front of the workspace)
  if (tid >= 128 * MT) {                       // the copying warps: a run's operands land while the runs before it are walked
    const int at = tid - 128 * MT;
    auto copy = [&](int c) {
      if (c < c_hi) {
        unsigned char* dst = csm + (c - c_lo) % stages * Z::STAGE;
        copy_bytes<QK_SIZE<D> * 2, COPY_THREADS<D>>(dst, reinterpret_cast<const unsigned char*>(qk + ((run0 + c) * G + g) * QK_SIZE<D>), at);
        dst += QK_SIZE<D> * 2;
        copy_bytes<PT_SIZE<false> * 2, COPY_THREADS<D>>(dst, reinterpret_cast<const unsigned char*>(pt + ((run0 + c) * H + h) * PT_SIZE<false>), at);
        float* dv = reinterpret_cast<float*>(dst + PT_SIZE<false> * 2);
#pragma unroll
        for (int e = at; e < RUN * 4 * MT; e += COPY_THREADS<D>) {
          const int t = e / (4 * MT), q = e % (4 * MT) * 4;
          const bool there = c * RUN + t < n;
          copy16(dv + t * Z::V_LD + q, x + (long long)(first + (there ? c * RUN + t : 0)) * C + voff + (long long)h * P + c0 + q, there);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    for (int i = 0; i < stages - 1; ++i) copy(c_lo + i);
    for (int c = c_lo; c < c_hi; ++c) {
      if (stages == 3) asm volatile("cp.async.wait_group 1;\n" ::);
      else asm volatile("cp.async.wait_group 0;\n" ::);
      __syncthreads();                           // run c is there; run c - 1 has been walked, and its stage is free
      copy(c + stages - 1);
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    return;
  }
  float4* red_q = reinterpret_cast<float4*>(csm + stages * Z::STAGE) + mt * (Z::MEET / 4);
  unsigned* ufr = reinterpret_cast<unsigned*>(red_q + 4 * RED);
  unsigned* efr = ufr + LEFT_WORDS;
  RunWarp<D> me;
  me.lane = lane; me.w = w; me.row = lane >> 2; me.two = (lane & 3) * 2;
  float* sp = state + (long long)slot * slot_stride + ((long long)h * P + c0 + mt * 16) * D + w * (D / 4);
  me.load(sp);
  me.terms();
  const float sk = skip[h];
  const long long ostride = (long long)H * P;
  float* op = out + (long long)first * ostride + (long long)h * P + c0 + mt * 16;
  const int row = me.row, t0 = w * 8 + me.two;   // this thread's tokens of a run: t0, t0 + 1
  for (int c = c_lo; c < c_hi; ++c) {
    __syncthreads();                             // the run's operands are there; what the last run put down has been read
    const bf16* dq = reinterpret_cast<const bf16*>(csm + (c - c_lo) % stages * Z::STAGE);
    const bf16* dk = dq + 3 * RUN * QK_LD<D>;
    const bf16* dp = dq + QK_SIZE<D>;
    const float* ds = reinterpret_cast<const float*>(dp + PLANE);
    const float* dv = ds + 2 * RUN + mt * 16;
    const float A0 = ds[t0], A1 = ds[t0 + 1], E0 = ds[RUN + t0], E1 = ds[RUN + t0 + 1], last = ds[RUN - 1];
    float v[4], e[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = dv[(t0 + (i & 1)) * Z::V_LD + row + 8 * (i >> 1)];
    const bool mine = not_finite(v);
    me.share(ufr, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = v[i] * (i & 1 ? E1 : E0);
    me.share(efr, e);
    me.against(dq, red_q);
    const bool odd = meet_any(1 + mt, mine);
    // S <- A_32 S + sum_s (E_s u_s) k_s^T for this warp's rows of state
    me.add(dk, efr, [&](int) { return make_float2(last, last); });
    me.terms();
    me.gather(o, red_q);
    // and what the run's own tokens give: the decayed q . k^T times u
    const int t = c * RUN + t0;
    float res[4];
    me.lower(res, dp, ufr);
    if (odd) lower_sums(res, dp, ufr, t0, row);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      res[i] = fmaf(i & 1 ? A1 : A0, o[i], res[i]);
      res[i] = fmaf(sk, v[i], res[i]);
    }
    if (t < n) {
      op[(long long)t * ostride + row] = res[0];
      op[(long long)t * ostride + row + 8] = res[2];
    }
    if (t + 1 < n) {
      op[(long long)(t + 1) * ostride + row] = res[1];
      op[(long long)(t + 1) * ostride + row + 8] = res[3];
    }
  }
  me.store(sp);
}

struct Args {
  const float *x, *decay, *weight, *skip;
  long long C;
  int qoff, koff, voff;
  const int *row_start, *row_slot;
  float* state;
  long long slot_stride;
  float* out;
  void* ws;
  int T, R, H, G, P, max_slots, max_q, min_tokens;
};

long long runs_of(int T, int R) { return (long long)T / RUN + R; }       // places for runs: see first_run

template <int D, bool DELTA> long long bytes_of(int H, int G) { return 2 * ((long long)G * QK_SIZE<D> + (long long)H * PT_SIZE<DELTA>); }
long long place_bytes(int H, int G, int D, bool delta) {
  return D == 64 ? (delta ? bytes_of<64, true>(H, G) : bytes_of<64, false>(H, G))
                 : (delta ? bytes_of<128, true>(H, G) : bytes_of<128, false>(H, G));
}

template <int D, int MT, bool DELTA> void walk(const Args& a, const bf16* qk, const bf16* pt, int lo, int hi, cudaStream_t stream) {
  const dim3 grid(a.P / (16 * MT), a.H, a.R);
  if constexpr (DELTA) {
    constexpr size_t smem = DeltaSmem<D, MT>::BYTES;
    raise_shared<chunk_delta_kernel<D, MT>>(smem);
    fmx_launch(chunk_delta_kernel<D, MT>, grid, dim3(128 * MT + 32), smem, stream, qk, pt, a.x, a.C, a.voff, a.row_start, a.row_slot, a.state,
               a.slot_stride, a.out, a.min_tokens, a.H, a.G, a.P, a.max_slots, lo, hi);
  } else {
    // three stages where a block has an SM to itself anyway
    using Z = PlainSmem<D, MT>;
    constexpr size_t most = Z::bytes(3) <= 227 * 1024 ? Z::bytes(3) : Z::bytes(2);
    const int stages = most > Z::bytes(2) && (long long)grid.x * a.H * a.R <= fmx_num_sms() ? 3 : 2;
    raise_shared<chunk_plain_kernel<D, MT>>(most);
    fmx_launch(chunk_plain_kernel<D, MT>, grid, dim3(128 * MT + COPY_THREADS<D>), Z::bytes(stages), stream, qk, pt, a.x, a.C, a.voff, a.skip, a.row_start,
               a.row_slot, a.state, a.slot_stride, a.out, a.min_tokens, a.H, a.G, a.P, a.max_slots, lo, hi, stages);
  }
}

// The step's runs in waves of `wave` places, whose operands the workspace holds; a state passes from wave to wave in its slot.
template <int D, bool DELTA> int launch(const Args& a, int wave, cudaStream_t stream) {
  bf16* qk = reinterpret_cast<bf16*>(a.ws);
  bf16* pt = qk + (long long)wave * a.G * QK_SIZE<D>;
  constexpr int prep = (2 * RUN * (D + 4) + (2 + PREP_WARPS<D>) * RUN * GRAM_LD) * 4;
  if (prep > 48 * 1024) raise_shared<chunk_prepare_kernel<D, DELTA>>(prep);
  // 32 columns a block halve the operands' traffic, at half as many blocks: with 128 rows of state, whose blocks of 16 fill an SM alone,
  // above one for each SM (512 tokens of each request, 32 heads of 64 values: 128 blocks 49 us and 66 with 32 columns, 256 82 and 68, 512 177
  // and 137), with 64 rows above two, where it costs up to a tenth at these sizes (384 87 and 90, 512 91 and 98, 1,024 177 and 196)
  const bool pair = a.P % 32 == 0 && (long long)a.R * a.H * (a.P / 16) > (long long)(D > 64 ? 1 : 2) * fmx_num_sms();
  const long long places = runs_of(a.T, a.R);
  for (long long at = 0; at < places; at += wave) {
    const int lo = (int)at, hi = (int)(at + wave < places ? at + wave : places);
    fmx_launch(chunk_prepare_kernel<D, DELTA>, dim3((a.max_q + RUN - 1) / RUN, a.G, a.R), dim3(32 * PREP_WARPS<D>), prep, stream, a.x, a.C, a.qoff,
               a.koff, a.decay, a.weight, 2 * a.H, a.row_start, a.min_tokens, a.H, a.G, qk, pt, lo, hi);
    if (pair) walk<D, 2, DELTA>(a, qk, pt, lo, hi, stream);
    else walk<D, 1, DELTA>(a, qk, pt, lo, hi, stream);
  }
  FMX_LAUNCH_CHECK();
  return 0;
}

int check(const char* who, const Args& a, int D, bool delta, long long ws_size) {
  if (a.T <= 0 || a.R <= 0 || a.H <= 0 || a.G <= 0 || a.H % a.G || a.P <= 0 || a.P % 16 || (D != 64 && D != 128) || a.max_q <= 0)
    return fmx_fail("%s: bad sizes T=%d R=%d H=%d G=%d D=%d P=%d max_q=%d", who, a.T, a.R, a.H, a.G, D, a.P, a.max_q);
  if (a.H > 65535 || a.R > 65535) return fmx_fail("%s: batch too large", who);
  if (a.C % 4 || a.slot_stride % 4 || (uintptr_t)a.x % 16 || (uintptr_t)a.state % 16 || (uintptr_t)a.ws % 16)
    return fmx_fail("%s: rows that do not start on 16 bytes", who);
  if (ws_size < place_bytes(a.H, a.G, D, delta)) return fmx_fail("%s: the workspace is too small", who);
  return 0;
}
int wave_of(const Args& a, int D, bool delta, long long ws_size) {      // places that a workspace holds
  const long long n = ws_size / place_bytes(a.H, a.G, D, delta), places = runs_of(a.T, a.R);
  return (int)(n < places ? n : places);
}
}  // namespace

// Bytes of workspace that T tokens of R rows take: all their runs, or as many as 256 MB hold (the rest follow in waves).
FMX_EXPORT long long fmx_chunk_scan_bytes(int T, int R, int H, int G, int D, int delta) {
  const long long one = place_bytes(H, G, D, delta != 0), places = runs_of(T, R), most = (256LL << 20) / one;
  return one * (places < most ? places : most < 1 ? 1 : most);
}

// The gated delta rule (see fmx_delta_rule) over the rows of at least min_tokens tokens; max_q: the longest one.
FMX_EXPORT int fmx_chunk_delta_rule(const float* qkv, const float* gb, const int* row_start, const int* row_slot, float* state,
                                    long long slot_stride, float* out, void* ws, long long ws_size, int T, int R, int H, int G,
                                    int D, int Dv, int max_slots, int max_q,
                                    int min_tokens, cudaStream_t stream) {
  const Args a = {qkv, gb, gb + H, nullptr, 2LL * G * D + (long long)H * Dv, 0, G * D, 2 * G * D, row_start, row_slot, state, slot_stride,
                  out, ws, T, R, H, G, Dv, max_slots, max_q, min_tokens};
  if (int bad = check("fmx_chunk_delta_rule", a, D, true, ws_size)) return bad;
  const int wave = wave_of(a, D, true, ws_size);
  return D == 64 ? launch<64, true>(a, wave, stream) : launch<128, true>(a, wave, stream);
}

// The state-space recurrence (see fmx_ssm_scan) over them.
FMX_EXPORT int fmx_chunk_ssm_scan(const float* xbc, const float* dd, const float* d_skip, const int* row_start, const int* row_slot,
                                  float* state, long long slot_stride, float* out, void* ws, long long ws_size, int T, int R, int H,
                                  int G, int N, int P, int max_slots, int max_q,
                                    int min_tokens, cudaStream_t stream) {
  const int inner = H * P;
  const Args a = {xbc, dd + H, dd, d_skip, (long long)inner + 2LL * G * N, inner + G * N, inner, 0, row_start, row_slot, state, slot_stride,
                  out, ws, T, R, H, G, P, max_slots, max_q, min_tokens};
  if (int bad = check("fmx_chunk_ssm_scan", a, N, false, ws_size)) return bad;
  const int wave = wave_of(a, N, false, ws_size);
  return N == 64 ? launch<64, false>(a, wave, stream) : launch<128, false>(a, wave, stream);
}
