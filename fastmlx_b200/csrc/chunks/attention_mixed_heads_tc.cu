// Tiled paged attention with sigmoid weights that are mixed across heads, for portions of prompts over a bfloat16 cache, on the
// tensor cores.  What it computes stands at the head of ../mixattn/attention_mixed_heads.cu, whose 32-bit multiply-adds
// it replaces where a tile holds enough tokens:
//
//     w_g(t, j) = sigmoid(cap(scale q_g(t) . k(j)) + b_g);   w'_h = sum_g M[h, g] w_g;   out_h(t) = sum_j w'_h(t, j) v(j)
//
// Keys and values are bfloat16; queries, weights, the mix and the mixed weights are 32-bit and enter their products as three
// bfloat16 terms (split_mma.cuh), so no product is rounded more than a 32-bit multiply-add rounds it.  An infinite score
// saturates its weight (`sum_of`); an infinite value, or an infinity in the mix, leaves NaN where 32-bit sums may leave an infinity.
//
// A block owns all heads of 8 tokens of one request and walks the keys in tiles of 32:
//   scores   two warps per key/value head: S^T = K Q^T, 32 keys by 8 tokens for each of a warp's two query heads; Q's
//            terms lie in shared memory as right fragments.  Cap and sigmoid; the weights go to shared memory as terms, rows of (key, token) per head.
//   mix      a warp per two keys: W = M P over all heads, terms back to where the keys' weights were.
//   values   two warps per key/value head again: O^T = V^T W^T, added to the registers' 32-bit sums tile by tile.
// The order of a sum over keys follows the number of blocks that share them out, and so the step's tokens and rows (fmx_mixattn_tc_plan).
// A row of 8 tokens is 16 bytes, so that every transposition is an ldmatrix.  Tokens are the products' 8 columns and keys,
// heads and value dimensions their 16 rows: with 16 tokens Q's terms and the weights
// would not fit shared memory.
//
// Per tile of 8 x 32 pairs 2,304 products, 4,700 cycles of the tensor pipe; it takes 12,000 (scores 2,400, sigmoids 2,150, mix
// 3,200, values 2,250, copies 1,600): bound by the phases' waits for one another.  Two query heads to a warp and Q's terms in
// shared memory: with four and Q in registers, eight warps of 255 registers took 14,900, sixteen with Q in registers spilled.
// One prompt of 1,531 tokens, 32 heads on 8 of 64 values: 825 us with 32-bit multiply-adds, 235 us here (2,048: 1,376 and 376);
// 64 tokens behind 2,000: 595 and 48 us.  Values that are not the bfloat16 nearest to 64-bit arithmetic's: 4.0e-4 and 1.7e-4.
#include <math.h>
#include <type_traits>
#include "split_mma.cuh"
#include "tanh_small.cuh"

namespace {
// At most KVH key heads of PER query heads of MAXD values: their 224 KB are what an SM has (Q's terms 96, keys and values 72, weights 50, the
// mix 6).  Larger sizes stay with 32-bit multiply-adds.
constexpr int TQ = 8, TK = 32, KVH = 8, PER = 4, HEADS = KVH * PER;
constexpr int WARPS = 16, HW = 2, THREADS = WARPS * 32;        // two warps to a key head, two query heads to a warp
constexpr int MAXD = 64, KLD = MAXD + 8;          // a key or value row in shared memory: eight rows' pieces meet no bank twice
constexpr int PROW = TK * TQ + 8;                 // a head's weights: 32 keys x 8 tokens, likewise
constexpr int PTERM = HEADS * PROW;
constexpr size_t MIX_BYTES = 3 * 2 * 2 * 32 * 16; // M as left fragments: term, 16 heads out, 16 heads in
constexpr size_t Q_BYTES = (size_t)HEADS * (MAXD / 16) * 3 * 32 * 8;            // Q as right fragments: head, 16 dimensions, term
constexpr size_t SMEM = (size_t)3 * PTERM * 2 + Q_BYTES + (size_t)2 * KVH * TK * KLD * 2 + MIX_BYTES + HEADS * 4;

__device__ __forceinline__ float ex2_approx(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// Places for the rows' tiles of 8 tokens: row r's first is row_start / 8 + r; rows do not overlap, whatever their lengths.
__global__ void __launch_bounds__(THREADS, 1)
mixed_heads_tc_kernel(const float* q, long long q_stride, const bf16* kv, const int* block_tables, int bt_stride, const int* positions,
                      const int* row_start, float* part, bf16* out, long long out_stride, int n_tokens, int nh, int nkv, int hd, int vd,
                      int page_size, long long num_pages, float scale, float softcap, int window, int R,
                      const float* __restrict__ head_bias, const float* __restrict__ mix, int min_tokens, int splits, int* status) {
  extern __shared__ __align__(16) unsigned char smem[];
  bf16* Ps = reinterpret_cast<bf16*>(smem);                 // [3][HEADS][PROW]: the weights, then in their place the mixed ones
  bf16* Ks = Ps + 3 * PTERM;                                // [KVH][TK][KLD]
  bf16* Vs = Ks + KVH * TK * KLD;
  uint4* Ms = reinterpret_cast<uint4*>(Vs + KVH * TK * KLD);
  uint2* Qs = reinterpret_cast<uint2*>(Ms + MIX_BYTES / 16);
  float* hb = reinterpret_cast<float*>(Qs + Q_BYTES / 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, two = (lane & 3) * 2, eight = lane >> 2;
  const int per = nh / nkv;
  const int kvh = warp >> 1, h0 = (warp & 1) * HW;          // a warp's key head, the first of its query heads
  const bool busy = kvh < nkv && h0 < per;
  auto slot_of = [&](int h) { return h / per * PER + h % per; };      // heads of a key/value head take slots of their own
  // ---- what needs nothing from the kernels before: the mix as fragments, the heads' numbers
  for (int e = tid; e < 3 * 2 * 2 * 32; e += THREADS) Ms[e] = make_uint4(0u, 0u, 0u, 0u);
  if (tid < HEADS) {
    const int c = tid / PER, hh = tid % PER;
    hb[tid] = c < nkv && hh < per && head_bias != nullptr ? head_bias[c * per + hh] : 0.f;
  }
  __syncthreads();
  bool small_terms = false;
  for (int e = tid; e < nh * nh; e += THREADS) {
    const int o = slot_of(e / nh), i = slot_of(e % nh);              // row (out), column (in)
    unsigned t[3];
    three_terms(mix[e], 0.f, t[0], t[1], t[2]);
    small_terms |= ((t[1] | t[2]) & 0x7fffu) != 0u;
    // left fragment of (row, column): register (row / 8 & 1) + 2 (column / 8 & 1), lane 4 (row % 8) + column % 8 / 2
    const int at = ((o >> 4) * 2 + (i >> 4)) * 32 + (o & 7) * 4 + ((i & 7) >> 1);
    const int reg = (o >> 3 & 1) + 2 * (i >> 3 & 1);
#pragma unroll
    for (int x = 0; x < 3; ++x)
      reinterpret_cast<bf16*>(Ms)[((x * 4 * 32 + at) * 4 + reg) * 2 + (i & 1)] = __ushort_as_bfloat16((unsigned short)(t[x] & 0xffffu));
  }
  // A mix that was stored in bfloat16 has no smaller terms: half of its products are with zeros and left out (the same
  // sums, bit for bit).  A whole layer of 1,531 tokens: 461 -> 454 us.
  const bool whole_mix = __syncthreads_or(small_terms) == 0;
  pdl_wait();
  pdl_trigger();
  // ---- this block's tokens
  const int place = (int)gridDim.x - 1 - (int)blockIdx.x, split = blockIdx.y;        // a row's last tiles walk the most keys: they start first
  int row = -1;
  for (int base = 0; base < R; base += THREADS)
    row += __syncthreads_count(base + tid < R && row_start[min(base + tid, R - 1)] / TQ + base + tid <= place);
  const int first = row_start[row], n_row = row_start[row + 1] - first;
  const int t0 = first + (place - (first / TQ + row)) * TQ;
  if (t0 >= first + n_row || n_row < min_tokens) return;
  const int n_q = min(TQ, first + n_row - t0);
  const int pos0 = positions[t0], pos_last = positions[t0 + n_q - 1];
  const int lo_min = window > 0 ? max(0, pos0 - window + 1) : 0;
  int kt = lo_min / TK, kt_end = pos_last >= 0 ? pos_last / TK + 1 : 0;
  {
    const int share = (max(0, kt_end - kt) + splits - 1) / splits;
    kt += split * share;
    kt_end = min(kt_end, kt + share);
  }
  // ---- Q's terms as right fragments: 16 dimensions, tokens across
  const int KT = hd >> 4, VT = vd >> 4;
  for (int e = tid; e < HEADS * (MAXD / 16) * 32; e += THREADS) {
    const int l = e & 31, k = e / 32 % (MAXD / 16), h = e / 32 / (MAXD / 16), c = h / PER, hh = h % PER;
    float2 a = make_float2(0.f, 0.f), b = a;
    if (c < nkv && hh < per && k < KT && (l >> 2) < n_q) {
      const float* p = q + (long long)(t0 + (l >> 2)) * q_stride + (long long)(c * per + hh) * hd + k * 16 + (l & 3) * 2;
      a = *reinterpret_cast<const float2*>(p);
      b = *reinterpret_cast<const float2*>(p + 8);
    }
    unsigned x[3], y[3];
    three_terms(a.x, a.y, x[0], x[1], x[2]);
    three_terms(b.x, b.y, y[0], y[1], y[2]);
#pragma unroll
    for (int t = 0; t < 3; ++t) Qs[((h * (MAXD / 16) + k) * 3 + t) * 32 + l] = make_uint2(x[t], y[t]);
  }
  float acc[HW][MAXD / 16][4];
#pragma unroll
  for (int hh = 0; hh < HW; ++hh)
#pragma unroll
    for (int m = 0; m < MAXD / 16; ++m)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[hh][m][i] = 0.f;
  // heads that are not there weigh nothing (their columns of the mix are zero, and so must their weights be: no NaN from old bits)
  for (int e = tid; e < 3 * PTERM / 2; e += THREADS) reinterpret_cast<unsigned*>(Ps)[e] = 0u;

  // ---- copies: a thread owns (key of the tile, 16-byte piece of a row) and walks the key/value heads.  A tile's page is looked
  // up a tile ahead: neither the division nor the load stands in front of a copy.
  const long long page_elems = (long long)nkv * page_size * (hd + vd);
  const int* bt = block_tables + (long long)row * bt_stride;
  const int jj = tid >> 3 & 31, ch = tid & 7, ch0 = tid >> 8;          // a thread takes every other key head from ch0 on
  struct Place { int page, at; };                           // page -2: out of sight
  auto look_up = [&](int tile) {
    Place l = {-2, 0};
    const int j = tile * TK + jj;
    if (tile < kt_end && j >= lo_min && j <= pos_last) {
      const int blk = j / page_size;
      l.at = j - blk * page_size;
      l.page = blk < bt_stride ? bt[blk] : -1;
    }
    return l;
  };
  auto copy = [&](Place l, bool there, bool values) {
    const int width = values ? vd : hd;
    if (there && ch * 8 < width) {
      const bf16* src = kv;
      unsigned bytes = 0;
      long long step = 0;
      if (l.page >= 0 && l.page < num_pages) {
        src = kv + (long long)l.page * page_elems + (values ? (long long)nkv * page_size * hd : 0) + (long long)l.at * width + ch * 8;
        step = (long long)page_size * width;
        bytes = 16;
      } else if (l.page != -2) {
        fmx_set_status(status, FMX_BAD_PAGE, l.page, t0);
      }
      unsigned sa = (unsigned)__cvta_generic_to_shared((values ? Vs : Ks) + jj * KLD + ch * 8);
#pragma unroll
      for (int c2 = 0; c2 < KVH; c2 += 2) {
        const int c = c2 + ch0;
        if (c < nkv)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa + c * TK * KLD * 2), "l"(src + c * step), "r"(bytes));
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  const float inv_cap = softcap > 0.f ? 1.0f / softcap : 0.f;
  unsigned* Pw = reinterpret_cast<unsigned*>(Ps);
  constexpr int WROW = PROW / 2, WTERM = PTERM / 2;         // in 32-bit words
  __syncthreads();
  Place here = look_up(kt), next = look_up(kt + 1);
  copy(here, kt < kt_end, false);
  for (; kt < kt_end; ++kt) {
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();                                        // the tile's keys are there; the values before it are read
    copy(here, true, true);
    // ---- scores
    if (busy) {
      const bf16* kc = Ks + kvh * TK * KLD;
      float s[2][HW][4], low[2][HW][4];                     // two tiles of 16 keys, two heads; sums of the leading and of the other terms
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int hh = 0; hh < HW; ++hh)
#pragma unroll
          for (int i = 0; i < 4; ++i) s[m][hh][i] = low[m][hh][i] = 0.f;
#pragma unroll
      for (int k = 0; k < MAXD / 16; ++k) {
        if (k >= KT) continue;
        unsigned a[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m) ldmatrix4(a[m], kc + (m * 16 + (lane & 15)) * KLD + k * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int hh = 0; hh < HW; ++hh) {
          const uint2* qp = Qs + ((kvh * PER + h0 + hh) * (MAXD / 16) + k) * 3 * 32 + lane;
          const uint2 q0 = qp[0], q1 = qp[32], q2 = qp[64];
#pragma unroll
          for (int m = 0; m < 2; ++m) mma16816(low[m][hh], a[m], q2.x, q2.y);
#pragma unroll
          for (int m = 0; m < 2; ++m) mma16816(s[m][hh], a[m], q0.x, q0.y);
#pragma unroll
          for (int m = 0; m < 2; ++m) mma16816(low[m][hh], a[m], q1.x, q1.y);
        }
      }
      // An infinity has no smaller terms (inf - inf), and one in a key meets queries' terms that are zero: where the sum is not finite,
      // the leading terms alone say what it is
      auto sum_of = [&](int m, int hh, int i) {
        const float all = s[m][hh][i] + low[m][hh][i];
        return all - all == 0.f ? all : s[m][hh][i];
      };
      if (softcap > 0.f) {
        bool large = false;
        const float to_y = scale * inv_cap;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int hh = 0; hh < HW; ++hh)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              s[m][hh][i] = sum_of(m, hh, i) * to_y;
              large |= fabsf(s[m][hh][i]) > TANH_SMALL;
            }
        if (__any_sync(0xffffffffu, large)) {
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int hh = 0; hh < HW; ++hh)
#pragma unroll
              for (int i = 0; i < 4; ++i) s[m][hh][i] = softcap * tanh_capped(s[m][hh][i]);
        } else {
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int hh = 0; hh < HW; ++hh)
#pragma unroll
              for (int i = 0; i < 4; ++i) s[m][hh][i] = softcap * tanh_small(s[m][hh][i]);
        }
      } else {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int hh = 0; hh < HW; ++hh)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[m][hh][i] = sum_of(m, hh, i) * scale;
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int key = m * 16 + eight, j = kt * TK + key;
        bool valid[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = two + (i & 1), jk = j + (i >> 1) * 8;
          valid[i] = jk <= pos0 + t && (window <= 0 || jk > pos0 + t - window) && t < n_q;
        }
#pragma unroll
        for (int hh = 0; hh < HW; ++hh) {
          if (h0 + hh >= per) continue;
          const int at = kvh * PER + h0 + hh;
          const float b = hb[at];
          float p[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) p[i] = valid[i] ? rcp_approx(1.0f + ex2_approx(-1.4426950408889634f * (s[m][hh][i] + b))) : 0.f;
          unsigned t[3], u[3];
          three_terms(p[0], p[1], t[0], t[1], t[2]);
          three_terms(p[2], p[3], u[0], u[1], u[2]);
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            unsigned* dst = Pw + x * WTERM + at * WROW + key * 4 + (lane & 3);
            dst[0] = t[x];
            dst[32] = u[x];
          }
        }
      }
    }
    __syncthreads();                                        // every head's weights are there; the keys are read
    copy(next, kt + 1 < kt_end, false);
    here = next;
    next = look_up(kt + 2);
    // ---- mix
    auto mix_keys = [&](auto whole) {
      constexpr int TERMS = decltype(whole)::value ? 1 : 3;              // of the mix
#pragma unroll
      for (int k2 = 0; k2 < TK / WARPS; k2 += 2) {            // two keys at a time: the mix's fragments are read once for both
        const int key = warp * (TK / WARPS) + k2;
        unsigned b[2][3][4];
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
          for (int x = 0; x < 3; ++x) ldmatrix4_trans(b[y][x], Ps + x * PTERM + lane * PROW + (key + y) * TQ);
        __syncwarp();                                         // read by all lanes: the mixed weights of these keys take their place
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
          for (int k = 0; k < 2; ++k) {
#pragma unroll
            for (int xa = TERMS - 1; xa >= 0; --xa) {         // one term of the mix at a time, the smallest first
              const uint4 v = Ms[((xa * 2 + m) * 2 + k) * 32 + lane];
              const unsigned a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int xb = 2 - xa; xb >= 0; --xb)
#pragma unroll
                for (int y = 0; y < 2; ++y) mma16816(xa + xb == 0 ? c[y] : d[y], a, b[y][xb][2 * k], b[y][xb][2 * k + 1]);
            }
          }
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            unsigned t[3], u[3];
            three_terms(c[y][0] + d[y][0], c[y][1] + d[y][1], t[0], t[1], t[2]);
            three_terms(c[y][2] + d[y][2], c[y][3] + d[y][3], u[0], u[1], u[2]);
#pragma unroll
            for (int x = 0; x < 3; ++x) {
              unsigned* dst = Pw + x * WTERM + (m * 16 + eight) * WROW + (key + y) * 4 + (lane & 3);
              dst[0] = t[x];
              dst[8 * WROW] = u[x];
            }
          }
        }
      }
    };
    if (whole_mix) mix_keys(std::true_type{});
    else mix_keys(std::false_type{});
    asm volatile("cp.async.wait_group 1;\n" ::);            // the values; the next tile's keys stay on their way
    __syncthreads();
    // ---- values
    if (busy) {
      const bf16* vc = Vs + kvh * TK * KLD;
      unsigned b[HW][3][4];
#pragma unroll
      for (int y = 0; y < HW; ++y)
#pragma unroll
        for (int x = 0; x < 3; ++x) ldmatrix4_trans(b[y][x], Ps + x * PTERM + (kvh * PER + h0 + y) * PROW + lane * TQ);
#pragma unroll
      for (int m = 0; m < MAXD / 16; ++m) {
        if (m >= VT) continue;
        unsigned a[2][4];
#pragma unroll
        for (int k = 0; k < 2; ++k)
          ldmatrix4_trans(a[k], vc + (k * 16 + (lane & 7) + (lane >> 4) * 8) * KLD + m * 16 + (lane >> 3 & 1) * 8);
        float c[HW][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int x = 2; x >= 0; --x)
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int y = 0; y < HW; ++y) mma16816(c[y], a[k], b[y][x][2 * k], b[y][x][2 * k + 1]);
#pragma unroll
        for (int y = 0; y < HW; ++y)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[y][m][i] += c[y][i];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  if (!busy) return;
#pragma unroll
  for (int hh = 0; hh < HW; ++hh) {
    if (h0 + hh >= per) continue;
#pragma unroll
    for (int m = 0; m < MAXD / 16; ++m) {
      if (m >= VT) continue;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = two + (i & 1), e = (kvh * per + h0 + hh) * vd + m * 16 + eight + (i >> 1) * 8;
        if (t >= n_q) continue;
        if (splits > 1) part[((long long)split * n_tokens + t0 + t) * nh * vd + e] = acc[hh][m][i];
        else out[(long long)(t0 + t) * out_stride + e] = __float2bfloat16_rn(acc[hh][m][i]);
      }
    }
  }
}

// The splits' parts in order; a block per token, tokens of rows that the kernel above left out stay.
__global__ void __launch_bounds__(256)
mixed_heads_tc_combine_kernel(const float* part, const int* token_row, const int* row_start, bf16* out, long long out_stride, int n_tokens,
                              int width, int R, int min_tokens, int splits) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, row = token_row[t];
  if (row < 0 || row >= R || row_start[row + 1] - row_start[row] < min_tokens) return;
  for (int x = threadIdx.x * 4; x < width; x += 1024) {
    float4 s = load4(part + (long long)t * width + x);
    for (int k = 1; k < splits; ++k) {
      const float4 v = load4(part + ((long long)k * n_tokens + t) * width + x);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    bf16* dst = out + (long long)t * out_stride + x;
    dst[0] = __float2bfloat16_rn(s.x); dst[1] = __float2bfloat16_rn(s.y);
    dst[2] = __float2bfloat16_rn(s.z); dst[3] = __float2bfloat16_rn(s.w);
  }
}

bool sizes_fit(int nh, int nkv, int hd, int vd) {
  return nkv > 0 && nkv <= KVH && nh > 0 && nh % nkv == 0 && nh / nkv <= PER && hd > 0 && hd <= MAXD && hd % 16 == 0 && vd > 0 && vd <= MAXD &&
         vd % 16 == 0;
}
}  // namespace

// How many blocks share out the keys of 8 tokens, or 0 where the kernel does not take the sizes.  A prompt's last tiles walk the
// most keys: with one block each they alone would run at the end (1,531 tokens: the longest of 192 walks 48 tiles, an
// SM's share is 31).  So many that the longest share is about an SM's; at least four tiles of keys to a block, and at most
// 256 MB of partial sums.  Behind a window (0: none) 8 tokens walk the tiles that window + 7 keys lie in.
FMX_EXPORT int fmx_mixattn_tc_plan(int n_tokens, int rows, int nh, int nkv, int hd, int vd, int max_q_len, int max_ctx, int window) {
  if (!sizes_fit(nh, nkv, hd, vd) || n_tokens <= 0) return 0;
  const long long tiles = n_tokens / TQ + rows, whole = (max_ctx + TK - 1) / TK;
  const long long held = window > 0 ? ((long long)window + TQ - 3) / TK + 2 : whole, longest = held < whole ? held : whole;
  const long long half = whole - max_q_len / 2 / TK, usual = half < longest ? half : longest;        // a row's tiles on average
  const long long total = tiles * (usual > 0 ? usual : 1);
  long long s = (longest * fmx_num_sms() + total - 1) / total;
  if (s > longest / 4) s = longest / 4;
  if (s > 32) s = 32;
  while (s > 1 && s * n_tokens * nh * vd * 4 > (256LL << 20)) --s;
  return s < 1 ? 1 : (int)s;
}

// As fmx_mixattn, for the rows of at least min_tokens tokens; part: splits * T * nh * vd floats where splits > 1.
FMX_EXPORT int fmx_mixattn_tc(const float* q, long long q_stride, const void* kv, const int* block_tables, int bt_stride,
                              const int* token_row, const int* positions, const int* row_start, float* part, void* out,
                              long long out_stride, int n_tokens, int nh, int nkv, int hd, int vd, int page_size, long long num_pages,
                              float scale, float softcap, int window, int R, const float* head_bias, const float* mix, int min_tokens,
                              int splits, int* status, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  if (n_tokens < 0 || R <= 0 || page_size <= 0 || window < 0 || splits < 1 || splits > 65535 || (splits > 1 && part == nullptr) || mix == nullptr)
    return fmx_fail("fmx_mixattn_tc: bad sizes T=%d R=%d page=%d window=%d splits=%d", n_tokens, R, page_size, window, splits);
  if (!sizes_fit(nh, nkv, hd, vd)) return fmx_fail("fmx_mixattn_tc: sizes nh=%d nkv=%d hd=%d vd=%d do not fit", nh, nkv, hd, vd);
  if (out_stride < (long long)nh * vd) return fmx_fail("fmx_mixattn_tc: output rows too narrow");
  if (((uintptr_t)q & 7) || (q_stride & 1) || ((uintptr_t)kv & 15) || (splits > 1 && ((uintptr_t)part & 15)))
    return fmx_fail("fmx_mixattn_tc: queries must lie on 8 bytes, pages and partial sums on 16");
  if (raise_shared<mixed_heads_tc_kernel>(SMEM) != cudaSuccess)
    return fmx_fail("fmx_mixattn_tc: the kernel's shared memory could not be raised");
  fmx_launch(mixed_heads_tc_kernel, dim3(n_tokens / TQ + R, splits), dim3(THREADS), SMEM, stream, q, q_stride, (const bf16*)kv, block_tables,
             bt_stride, positions, row_start, part, (bf16*)out, out_stride, n_tokens, nh, nkv, hd, vd, page_size, num_pages, scale, softcap,
             window, R, head_bias, mix, min_tokens, splits, status);
  if (splits > 1)
    fmx_launch(mixed_heads_tc_combine_kernel, dim3(n_tokens), dim3(256), 0, stream, (const float*)part, token_row, row_start, (bf16*)out,
               out_stride, n_tokens, nh * vd, R, min_tokens, splits);
  FMX_LAUNCH_CHECK();
  return 0;
}
