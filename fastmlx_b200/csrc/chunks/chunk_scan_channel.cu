// Linear recurrences whose state decays by key channel, over portions, in runs of 32 tokens as matrix products:
//
//     S <- diag(a_t) S + k_t u_t^T;   o_t = S^T q_t;   u_t = v_t, or the delta rule's u_t = beta_t (v_t - (diag(a_t) S)^T k_t)
//
// with a decay per head and row of S.  The same form as chunk_scan.cu, with A_t = a_1 ... a_t a vector and on the operands:
//
//     o_t = S^T (A_t q_t) + sum_{s <= t} P_ts u_s,                P_ts = sum_d q_td k_sd (A_t / A_s)_d
//     u   = T diag(beta) (v - S^T (A_t k_t)),                     T = (1 + strictly lower part of beta_t sum_d k_td k_sd (A_t / A_s)_d)^-1
//     S  <- diag(A_32) S + sum_s ((A_32 / A_s) k_s) u_s^T
//
// Ratios are running products of decays, in P and T too: a ratio of two products of 32 decays would be 0 / 0 where a channel
// forgets quickly.  So P and T are 32-bit multiply-adds (a k_s decays as t goes on, as in the walk token by token) and
// everything that meets the state runs on the tensor cores with three bfloat16 terms an operand (split_mma.cuh).
//
//   channel_prepare   per (run, head): P, T, and A q, A k, (A_32 / A) k as three terms.  All runs of a wave at once.
//   channel_chunks    per (request, head, 16 or 32 columns of S): the runs in order.
//
// The operands of a run and head are 57 KB (64 rows of state) or 94 KB (128), so a step's runs go in waves whose workspace is
// bounded.  An infinity or a NaN reaches what it reaches in chunk_scan.cu.
// 32 heads on 8 key heads of 128 x 128, 2,048 tokens: one request 754 us token by token and 342 here, two of 768 and 1,280 637 and 352
// (of which 150 to prepare and 199 for the runs).  64 x 64, one request: 387 and 249; without the delta rule 265 and 204, while 128 x 128
// takes 308 either way and stays with the walk.  Against 64-bit: 1.3e-7 of the result's norm, 1.4e-7 token by token.
#include <math.h>
#include "runs.cuh"

namespace {
template <int D> constexpr int K_LD = D + 8;
template <int D> constexpr int K_PLANE = 3 * RUN * K_LD<D>;                   // bf16 of one 32 x D matrix in three terms
// a run and head: in front A k (delta rule) and A q; behind them (A_32 / A) k, P, T (delta rule) and, as floats, A_32
template <int D, bool DELTA> constexpr int FRONT = (DELTA ? 2 : 1) * K_PLANE<D>;
template <int D, bool DELTA> constexpr int BACK = K_PLANE<D> + (DELTA ? 2 : 1) * PLANE + 2 * D;

struct ChannelArgs {
  const float *qkv, *decay, *beta;             // [T, C], [T, H D], [T, H]
  const int *row_start, *row_slot;
  float* state;
  long long slot_stride;
  float* out;
  bf16* ws;
  int R, H, G, P, max_slots, min_tokens;
  int lo, hi;                                  // the wave's places; row r's runs take places from row_start / 32 + r on
};

// a 32 x N matrix of floats (rows LD apart) as three terms (rows OUT_LD apart), by `threads` threads from `tid` on
template <int N, int LD, int OUT_LD> __device__ __forceinline__ void emit_terms(const float* src, bf16* dst, int tid, int threads) {
#pragma unroll 4
  for (int e = tid; e < RUN * (N / 4); e += threads) {
    const int row = e / (N / 4), c = e % (N / 4) * 4;
    const float4 v = load4(src + row * LD + c);
    unsigned a[3], b[3];
    three_terms(v.x, v.y, a[0], a[1], a[2]);
    three_terms(v.z, v.w, b[0], b[1], b[2]);
#pragma unroll
    for (int t = 0; t < 3; ++t) *reinterpret_cast<uint2*>(dst + (t * RUN + row) * OUT_LD + c) = make_uint2(a[t], b[t]);
  }
}

// Eight warps: a lane holds a token's k, a warp an eighth of the channels, and as t goes on a lane's k decays and meets q_t and k_t,
// which all lanes read together; no sum crosses lanes, the warps' shares are added up in order.  Bound by the latency of a
// block's phases (with four warps a run and head took twice as long), of which two blocks share an SM.
constexpr int PREP_THREADS = 256, PREP_WARPS = 8;
template <int D> constexpr int PREP_SMEM = (3 * RUN * (D + 4) + (PREP_WARPS + 2) * RUN * GRAM_LD) * 4;

template <int D, bool DELTA>
__global__ void __launch_bounds__(PREP_THREADS)
channel_prepare_kernel(ChannelArgs a) {
  constexpr int LD = D + 4, DS = D / PREP_WARPS;
  extern __shared__ __align__(16) float psm[];
  float* qs = psm;                             // [32][LD]; then A q
  float* ks = qs + RUN * LD;
  float* gs = ks + RUN * LD;
  float* pm = gs + RUN * LD;                   // [P, M][32][GRAM_LD]
  float* part = pm + 2 * RUN * GRAM_LD;        // [8 warps][P, M][16][GRAM_LD]; then (A_32 / A) k | A k, [32][LD] each
  static_assert(2 * LD <= PREP_WARPS * GRAM_LD, "both fit");
  const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int place = a.lo + (int)blockIdx.x;
  pdl_wait();
  int r = -1;
  for (int base = 0; base < a.R; base += PREP_THREADS)
    r += __syncthreads_count(base + tid < a.R && a.row_start[min(base + tid, a.R - 1)] / RUN + base + tid <= place);
  const int first = a.row_start[r], n = a.row_start[r + 1] - first, c = place - (first / RUN + r);
  if (c * RUN >= n || n < a.min_tokens) return;
  const int t0 = first + c * RUN, cnt = min(RUN, n - c * RUN), g = h / (a.H / a.G);
  const long long C = 2LL * a.G * D + (long long)a.H * a.P;
#pragma unroll 4
  for (int e = tid; e < 3 * RUN * (D / 4); e += PREP_THREADS) {
    const int which = e / (RUN * (D / 4)), row = e / (D / 4) % RUN, d = e % (D / 4) * 4;
    float4 v = which == 2 ? make_float4(1.f, 1.f, 1.f, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < cnt) v = which == 2 ? load4(a.decay + (long long)(t0 + row) * a.H * D + (long long)h * D + d)
                                  : load4(a.qkv + (long long)(t0 + row) * C + (long long)(which * a.G + g) * D + d);
    store4((which == 0 ? qs : which == 1 ? ks : gs) + row * LD + d, v);
  }
  const float beta = DELTA && lane < cnt ? a.beta[(long long)(t0 + lane) * a.H + h] : 0.f;       // of token `lane`
  __syncthreads();
  f32x2 kd[DS / 2];                            // this lane's token's k, decayed to the token t
#pragma unroll
  for (int i = 0; i < DS; i += 4) {
    const float4 v = load4(ks + lane * LD + warp * DS + i);
    kd[i / 2] = pair_of(v.x, v.y);
    kd[i / 2 + 1] = pair_of(v.z, v.w);
  }
#pragma unroll 1
  for (int t1 = 0; t1 < RUN; t1 += 16) {       // sixteen tokens' shares at a time
#pragma unroll 2
    for (int t = t1; t < t1 + 16; ++t) {
      const ulonglong2* gt = reinterpret_cast<const ulonglong2*>(gs + t * LD + warp * DS);
      const ulonglong2* qt = reinterpret_cast<const ulonglong2*>(qs + t * LD + warp * DS);
      const ulonglong2* kt = reinterpret_cast<const ulonglong2*>(ks + t * LD + warp * DS);
      ulonglong2 gv[DS / 4], qv[DS / 4], kv[DS / 4];
#pragma unroll
      for (int i = 0; i < DS / 4; ++i) {
        gv[i] = gt[i];
        qv[i] = qt[i];
        if (DELTA) kv[i] = kt[i];
      }
      if (lane < t) {
#pragma unroll
        for (int i = 0; i < DS / 4; ++i) {
          kd[2 * i] = mul2(kd[2 * i], gv[i].x);
          kd[2 * i + 1] = mul2(kd[2 * i + 1], gv[i].y);
        }
      }
      f32x2 p[2] = {0ull, 0ull}, m[2] = {0ull, 0ull};
#pragma unroll
      for (int i = 0; i < DS / 4; ++i) {
        p[0] = fma2(kd[2 * i], qv[i].x, p[0]);
        p[1] = fma2(kd[2 * i + 1], qv[i].y, p[1]);
        if (DELTA) {
          m[0] = fma2(kd[2 * i], kv[i].x, m[0]);
          m[1] = fma2(kd[2 * i + 1], kv[i].y, m[1]);
        }
      }
      part[(warp * 32 + t - t1) * GRAM_LD + lane] = pair_sum(p[0]) + pair_sum(p[1]);
      if (DELTA) part[(warp * 32 + 16 + t - t1) * GRAM_LD + lane] = pair_sum(m[0]) + pair_sum(m[1]);
    }
    __syncthreads();
    // the warps' shares; P up to t = s, M (times beta_t) up to t = s + 1; a warp takes a row
    for (int e = warp; e < (DELTA ? 32 : 16); e += PREP_WARPS) {
      const int which = e >> 4, t = t1 + (e & 15);
      const float* src = part + e * GRAM_LD + lane;
      float s[PREP_WARPS];
#pragma unroll
      for (int i = 0; i < PREP_WARPS; ++i) s[i] = src[i * 32 * GRAM_LD];
      float v = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
      if (which) v *= __shfl_sync(0xffffffffu, beta, t);
      pm[(which * RUN + t) * GRAM_LD + lane] = (which ? lane < t : lane <= t) ? v : 0.f;
    }
    __syncthreads();
  }
  bf16* front = a.ws + ((long long)blockIdx.x * a.H + h) * (FRONT<D, DELTA> + BACK<D, DELTA>);
  bf16* back = front + FRONT<D, DELTA>;
  if (DELTA && warp == 0) {
    float* M = pm + RUN * GRAM_LD;
    solve_unit_lower(M, lane, beta);
    emit_terms<RUN, GRAM_LD, PT_LD>(M, back + K_PLANE<D> + PLANE, lane, 32);
    return;
  }
  constexpr int threads = DELTA ? PREP_THREADS - 32 : PREP_THREADS;
  const int at = DELTA ? tid - 32 : tid;
  float *ke = part, *ka = part + RUN * LD;
  float* last = reinterpret_cast<float*>(back + K_PLANE<D> + (DELTA ? 2 : 1) * PLANE);
  for (int x = at; x < 2 * D; x += threads) {  // a column each: the decays behind a token, or those up to it
    const int d = x < D ? x : x - D;
    float e = 1.f;
    if (x < D) {
#pragma unroll 16
      for (int t = RUN - 1; t >= 0; --t) {
        ke[t * LD + d] = ks[t * LD + d] * e;
        e *= gs[t * LD + d];
      }
    } else {
#pragma unroll 16
      for (int t = 0; t < RUN; ++t) {
        e *= gs[t * LD + d];
        qs[t * LD + d] *= e;
        if (DELTA) ka[t * LD + d] = ks[t * LD + d] * e;
      }
      last[d] = e;
    }
  }
  if (DELTA) asm volatile("bar.sync 1, 224;\n" ::: "memory");
  else __syncthreads();
  if (DELTA) emit_terms<D, LD, K_LD<D>>(ka, front, at, threads);
  emit_terms<D, LD, K_LD<D>>(qs, front + (DELTA ? K_PLANE<D> : 0), at, threads);
  emit_terms<D, LD, K_LD<D>>(ke, back, at, threads);
  emit_terms<RUN, GRAM_LD, PT_LD>(pm, back + K_PLANE<D>, at, threads);
}

template <int D, int MT, bool DELTA> struct ChannelSmem {
  static constexpr int V_LD = 16 * MT + 4;
  static constexpr size_t FRONT_BYTES = (size_t)FRONT<D, DELTA> * 2 + (size_t)RUN * V_LD * 4, BACK_BYTES = (size_t)BACK<D, DELTA> * 2;
  static constexpr int S_WORDS = 3 * (D / 16) * 32 * 4, U_WORDS = 3 * (RUN / 16) * 32 * 4;
  static constexpr size_t BYTES = FRONT_BYTES + BACK_BYTES + (size_t)MT * (S_WORDS + (DELTA ? 2 : 1) * U_WORDS) * 4;
};

// Threads that copy: with 128 rows of state, whose block fills an SM, four warps, since everything waits for the copies (two prompts of 768 and
// 1,280 tokens, 32 heads: 227 us with one, 199 with four); with 64 rows the registers of a second warp cost more than it brings (three requests of
// 512 tokens 114 and 140 us).
template <int D> constexpr int CHANNEL_COPY = D > 64 ? 128 : 32;

// As chunk_delta_kernel (four warps per 16 columns, others that copy), but a run's operands are twice as many bytes: one buffer for what
// the state is multiplied with in front and one for what comes after, each filled while the other one is in use.
template <int D, int MT, bool DELTA>
__global__ void __launch_bounds__(128 * MT + CHANNEL_COPY<D>)
channel_chunks_kernel(ChannelArgs a) {
  using Z = ChannelSmem<D, MT, DELTA>;
  constexpr int KT = D / 16, NS = D / 32, QK_LD = K_LD<D>;
  extern __shared__ __align__(16) unsigned char csm[];
  const int r = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * 16 * MT;
  const int tid = threadIdx.x, lane = tid & 31, mt = tid >> 7, w = tid >> 5 & 3;
  pdl_wait();
  pdl_trigger();
  const int slot = a.row_slot[r];
  if (slot < 0 || slot >= a.max_slots) return;
  const int first = a.row_start[r], n = a.row_start[r + 1] - first;
  if (n < a.min_tokens) return;
  const int base = first / RUN + r;            // the row's runs of this wave
  const int lo = max(0, a.lo - base), hi = min((n + RUN - 1) / RUN, a.hi - base);
  if (lo >= hi) return;
  const long long C = 2LL * a.G * D + (long long)a.H * a.P;
  bf16* fr = reinterpret_cast<bf16*>(csm);
  float* dv = reinterpret_cast<float*>(fr + FRONT<D, DELTA>);
  bf16* bk = reinterpret_cast<bf16*>(csm + Z::FRONT_BYTES);
  if (tid >= 128 * MT) {                       // the copying warps
    const int at = CHANNEL_COPY<D> == 32 ? lane : tid - 128 * MT;
    auto landed = []() {
      asm volatile("cp.async.commit_group;\n" ::);
      asm volatile("cp.async.wait_group 0;\n" ::);
    };
    const float* vp = a.qkv + 2LL * a.G * D + (long long)h * a.P + c0;
    for (int c = lo; c < hi; ++c) {
      const unsigned char* src = reinterpret_cast<const unsigned char*>(a.ws + ((long long)(base + c - a.lo) * a.H + h) * (FRONT<D, DELTA> + BACK<D, DELTA>));
      copy_bytes<FRONT<D, DELTA> * 2, CHANNEL_COPY<D>>(csm, src, at);
#pragma unroll
      for (int e = at; e < RUN * 4 * MT; e += CHANNEL_COPY<D>) {
        const int t = e / (4 * MT), q = e % (4 * MT) * 4;
        const bool there = c * RUN + t < n;
        copy16(dv + t * Z::V_LD + q, vp + (long long)(first + (there ? c * RUN + t : 0)) * C + q, there);
      }
      landed();
      __syncthreads();                         // (1) run c's front is there, the back of run c - 1 has been read
      copy_bytes<BACK<D, DELTA> * 2, CHANNEL_COPY<D>>(csm + Z::FRONT_BYTES, src + FRONT<D, DELTA> * 2, at);
      landed();
      __syncthreads_or(0);                     // (2) its back is there, its front has been read
    }
    return;
  }
  unsigned* sfr = reinterpret_cast<unsigned*>(csm + Z::FRONT_BYTES + Z::BACK_BYTES) + mt * Z::S_WORDS;
  unsigned* ufr = reinterpret_cast<unsigned*>(csm + Z::FRONT_BYTES + Z::BACK_BYTES) + MT * Z::S_WORDS + mt * (DELTA ? 2 : 1) * Z::U_WORDS;
  unsigned* rfr = ufr + Z::U_WORDS;
  const int row = lane >> 2, two = (lane & 3) * 2;
  float* sp = a.state + (long long)slot * a.slot_stride + ((long long)h * a.P + c0 + mt * 16) * D + w * (D / 4);
  float S[NS][4];
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const float2 x = *reinterpret_cast<const float2*>(sp + (long long)row * D + j * 8 + two);
    const float2 y = *reinterpret_cast<const float2*>(sp + (long long)(row + 8) * D + j * 8 + two);
    S[j][0] = x.x; S[j][1] = x.y; S[j][2] = y.x; S[j][3] = y.y;
  }
  auto share_state = [&]() {
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
  auto share_tile = [&](unsigned* dst, const float (&v)[4]) {
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
  const long long ostride = (long long)a.H * a.P;
  float* op = a.out + (long long)first * ostride + (long long)h * a.P + c0 + mt * 16;
  const int t0 = w * 8 + two, rows8 = w * 8 + (lane & 7), quarter = (lane >> 3) * 8;
  const bf16* dq = fr + (DELTA ? K_PLANE<D> : 0);
  const bf16* dp = bk + K_PLANE<D>;
  const float* last = reinterpret_cast<const float*>(dp + (DELTA ? 2 : 1) * PLANE) + w * (D / 4) + two;
  for (int c = lo; c < hi; ++c) {
    __syncthreads();                           // (1)
    const float* v0 = dv + mt * 16;
    float v[4] = {v0[t0 * Z::V_LD + row], v0[(t0 + 1) * Z::V_LD + row], v0[t0 * Z::V_LD + row + 8], v0[(t0 + 1) * Z::V_LD + row + 8]};
    Sums o, kS;
    o.zero();
    kS.zero();
#pragma unroll
    for (int k2 = 0; k2 < KT / 2; ++k2) {
      unsigned bq[3][4], bkk[3][4];
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        if (DELTA) ldmatrix4(bkk[t], fr + (t * RUN + rows8) * QK_LD + k2 * 32 + quarter);
        ldmatrix4(bq[t], dq + (t * RUN + rows8) * QK_LD + k2 * 32 + quarter);
      }
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        unsigned f[3][4];
        fragment(f, sfr, KT, k2 * 2 + kk);
        if (DELTA) kS.add(f, bkk, kk * 2);
        o.add(f, bq, kk * 2);
      }
    }
    if (DELTA) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] -= kS.at(i);
      share_tile(rfr, v);
    } else {
      share_tile(ufr, v);
    }
    bool odd = __syncthreads_or(not_finite(v));        // (2)
    if (DELTA) {                               // u = T diag(beta) (v - (A k) S)
      unsigned bt[3][4];
      Sums u;
      u.zero();
#pragma unroll
      for (int t = 0; t < 3; ++t) ldmatrix4(bt[t], dp + PLANE + (t * RUN + rows8) * PT_LD + quarter);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (k <= (w >> 1)) {
          unsigned f[3][4];
          fragment(f, rfr, 2, k);
          u.add(f, bt, k * 2);
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = u.at(i);
      if (odd) lower_sums(v, dp + PLANE, rfr, t0, row);
      const bool mine = not_finite(v);
      share_tile(ufr, v);
      odd = meet_any(1 + mt, mine);
    }
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
        unsigned f[3][4];
        fragment(f, ufr, 2, k);
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          unsigned b[3][2];
#pragma unroll
          for (int t = 0; t < 3; ++t) ldmatrix2_trans(b[t], bk + (t * RUN + k * 16 + (lane & 15)) * QK_LD + w * (D / 4) + j * 8);
          d[j].add(f, b, 0);
        }
        if (k <= (w >> 1)) y.add(f, bp, k * 2);
      }
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      const float2 e = *reinterpret_cast<const float2*>(last + j * 8);
      S[j][0] = fmaf(S[j][0], e.x, d[j].at(0)); S[j][1] = fmaf(S[j][1], e.y, d[j].at(1));
      S[j][2] = fmaf(S[j][2], e.x, d[j].at(2)); S[j][3] = fmaf(S[j][3], e.y, d[j].at(3));
    }
    share_state();                             // the others' reads of these fragments lie in front of (2)
    const int t = c * RUN + t0;
    float res[4] = {y.at(0), y.at(1), y.at(2), y.at(3)};
    if (odd) lower_sums(res, dp, ufr, t0, row);
#pragma unroll
    for (int i = 0; i < 4; ++i) res[i] += o.at(i);
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

template <int D, bool DELTA> int launch(ChannelArgs a, int places, int per_wave, cudaStream_t stream) {
  constexpr int prep = PREP_SMEM<D>;
  raise_shared<channel_prepare_kernel<D, DELTA>>(prep);
  // 32 columns a block as in chunk_scan.cu, above one (128 rows) and three (64 rows) blocks of 16 for each SM.  At 512 tokens of each
  // request, 32 heads of 64 values, that is no gain: 128 rows 384 blocks 238 us and 244, 1,024 573 and 594; 64 rows 512 181 and 192, 1,024 319
  // and 380 (without the delta rule 512 137 and 144).
  const bool pair = a.P % 32 == 0 && (long long)a.R * a.H * (a.P / 16) > (long long)(D > 64 ? 1 : 3) * fmx_num_sms();
  for (a.lo = 0; a.lo < places; a.lo += per_wave) {
    a.hi = a.lo + per_wave < places ? a.lo + per_wave : places;
    fmx_launch(channel_prepare_kernel<D, DELTA>, dim3(a.hi - a.lo, a.H), dim3(PREP_THREADS), prep, stream, a);
    if (pair) {
      constexpr size_t smem = ChannelSmem<D, 2, DELTA>::BYTES;
      raise_shared<channel_chunks_kernel<D, 2, DELTA>>(smem);
      fmx_launch(channel_chunks_kernel<D, 2, DELTA>, dim3(a.P / 32, a.H, a.R), dim3(256 + CHANNEL_COPY<D>), smem, stream, a);
    } else {
      constexpr size_t smem = ChannelSmem<D, 1, DELTA>::BYTES;
      raise_shared<channel_chunks_kernel<D, 1, DELTA>>(smem);
      fmx_launch(channel_chunks_kernel<D, 1, DELTA>, dim3(a.P / 16, a.H, a.R), dim3(128 + CHANNEL_COPY<D>), smem, stream, a);
    }
  }
  FMX_LAUNCH_CHECK();
  return 0;
}

long long place_bytes(int H, int D, bool delta) {
  return 2LL * H * (!delta ? FRONT<64, false> + BACK<64, false> : D == 64 ? FRONT<64, true> + BACK<64, true> : FRONT<128, true> + BACK<128, true>);
}
}  // namespace

// Bytes of workspace that T tokens of R rows take: all their runs, or as many as 256 MB hold (the rest follow in waves).
FMX_EXPORT long long fmx_channel_chunks_bytes(int T, int R, int H, int D, int delta) {
  const long long one = place_bytes(H, D, delta != 0), places = (long long)T / RUN + R, most = (256LL << 20) / one;
  return one * (places < most ? places : most < 1 ? 1 : most);
}

// The recurrence of fmx_channel_scan (beta null: without the delta rule) over the rows of at least min_tokens tokens.
FMX_EXPORT int fmx_channel_chunks(const float* qkv, const float* decay, const float* beta, const int* row_start, const int* row_slot,
                                  float* state, long long slot_stride, float* out, void* ws, long long ws_size, int T, int R, int H, int G,
                                  int D, int Dv, int max_slots, int min_tokens, cudaStream_t stream) {
  if (T <= 0 || R <= 0 || H <= 0 || G <= 0 || H % G || Dv <= 0 || Dv % 16 || (D != 64 && (D != 128 || beta == nullptr)))
    return fmx_fail("fmx_channel_chunks: bad sizes T=%d R=%d H=%d G=%d D=%d Dv=%d", T, R, H, G, D, Dv);
  if (H > 65535 || R > 65535) return fmx_fail("fmx_channel_chunks: batch too large");
  if (slot_stride % 4 || (uintptr_t)qkv % 16 || (uintptr_t)decay % 16 || (uintptr_t)state % 16 || (uintptr_t)ws % 16)
    return fmx_fail("fmx_channel_chunks: rows that do not start on 16 bytes");
  const long long per_wave = ws_size / place_bytes(H, D, beta != nullptr), places = (long long)T / RUN + R;
  if (per_wave < 1) return fmx_fail("fmx_channel_chunks: the workspace is too small");
  const ChannelArgs a = {qkv, decay, beta, row_start, row_slot, state, slot_stride, out, (bf16*)ws, R, H, G, Dv, max_slots, min_tokens, 0, 0};
  const int wave = (int)(per_wave < places ? per_wave : places);
  if (beta == nullptr) return launch<64, false>(a, (int)places, wave, stream);
  return D == 64 ? launch<64, true>(a, (int)places, wave, stream) : launch<128, true>(a, (int)places, wave, stream);
}
