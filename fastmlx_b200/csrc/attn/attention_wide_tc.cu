// Paged causal attention with 32-bit queries, two-term products and optionally a window and capped scores, for portions of prompts, on the
// fifth-generation tensor cores (head sizes 64 and 128; compile with -DFMX_HD=<head size>).  What it computes is the second form
// of the prefill kernel of attention_bf16.cu: queries and weights enter their products as two bfloat16 terms (16 bits of mantissa),
// sums are 32-bit, s <- cap tanh(s / cap) in front of the softmax.
//
// A CTA owns one or two tiles of 128 packed query rows of one request and kv head (row i: token i / rep, query head g rep + i % rep),
// which share the key and value tiles.
//   warp 0     brings key and value tiles, a page at a time by TMA; pages out of sight read as zeros.
//   warp 1     issues the products: S = Q1 K^T + Q2 K^T into tensor memory, O += P2 V + P1 V with P read from there.
//   the others a softmax group of four warps per query tile, a thread per row: the row's maximum, then its weights, whose leading
//              terms replace the scores; the output is rescaled only where a row's maximum has grown by more than 2^8.
// Two score buffers per query tile: the next scores are there when a group is done with the last ones, and a tile's output
// product runs beside the next tile's softmax.
// Bound by the softmax's arithmetic (the capping polynomial and the split of the weights, in packed pairs) and, behind it, by the products.
// Against the `mma.sync` kernel, 2,499 tokens of three portions behind 700, 32 heads on 8, us: head size 64, window 1,024 and capped
// scores 168 -> 81, neither 155 -> 74; head size 128 295 -> 121 and 293 -> 123.  On the way there, for the first of these: one score buffer
// and tiles of 128 keys 141, two buffers 115, one query tile a CTA 102, the polynomial in packed pairs 85, sums and split too 81.
// Every wait is bounded by time; one that runs out leaves FMX_WAIT_EXPIRED in the status word.
#include <type_traits>
#include "packed.cuh"
#include "tanh_small.cuh"
#include "tcgen05.cuh"

#ifndef FMX_HD
#error "compile with -DFMX_HD=<head size>"
#endif

#if FMX_HD == 64 || FMX_HD == 128
namespace {
using namespace fmx_tc;
constexpr int HD = FMX_HD, KB = HD / 64;       // 64-wide blocks of the head dimension
constexpr int BM = 128, BN = 64;               // query rows, keys of a tile
// Query tiles of a CTA.  At head size 64 one, and two CTAs share an SM: half as much work a CTA fills the GPU's rounds better
// (115 -> 102 us, see above); at 128 the second CTA would not fit.
constexpr int NX = HD == 64 ? 1 : 2;
constexpr int BLOCK = 128 * 128;               // a [128 x 64] bfloat16 block, 128-byte rows
constexpr int Q_TERM = KB * BLOCK, Q_TILE = 2 * Q_TERM;
constexpr int KV_HALF = KB * BN * 128, KV_BYTES = 2 * KV_HALF;     // a tile's keys, then its values
constexpr int STAGES = HD == 64 ? 4 : 3;
constexpr int THREADS = 64 + 128 * NX;
constexpr int S_COL = 0, O_COL = 2 * NX * BN;       // two score buffers a query tile
constexpr int TMEM_COLS = 256 * NX;
static_assert(O_COL + NX * HD <= TMEM_COLS, "scores and outputs must fit tensor memory");
constexpr size_t SMEM = NX * (size_t)Q_TILE + (size_t)STAGES * KV_BYTES + 1024 + 256;
constexpr float LOG2E = 1.4426950408889634f;

struct Wide {
  const float* q;
  long long q_stride;
  const int *block_tables, *row_start, *row_ctx, *positions;
  bf16* out;
  long long out_stride, num_pages, kv_rows;
  int bt_stride, nh, nkv, page_size, window;
  float scale, softcap;
  int out16;
  int* status;
};

struct WideBars {
  uint64_t kv_full[STAGES], kv_empty[STAGES];
  uint64_t s_full[NX][2], p_full[NX][2], pv_done[NX][2];      // per query tile and score buffer
  uint32_t tmem_slot;
};

__device__ __forceinline__ float exp2_fast(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ void two_terms(float x, float y, unsigned& hi, unsigned& lo) {
  hi = pack2(x, y);
  lo = pack2(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}
// tanh y = y + y^3 P(y^2) for |y| <= TANH_SMALL, P of degree five fitted to it there (largest error 1.5e-9, in 32-bit arithmetic 5.1e-8):
// multiply-adds and no reciprocal, of which the special-function unit has enough to do with the exponentials.
__device__ __forceinline__ float tanh_short(float y) {
  const float q = y * y;
  float p = fmaf(q, 0.00152817f, -0.00729639f);
  p = fmaf(q, p, 0.02121742f);
  p = fmaf(q, p, -0.05382224f);
  p = fmaf(q, p, 0.13331741f);
  p = fmaf(q, p, -0.33333272f);
  return fmaf(y * q, p, y);
}
// The same for two scores in packed multiply-adds, which round alike.
__device__ __forceinline__ f32x2 tanh_short(f32x2 y) {
  auto both = [](float c) { return pair_of(c, c); };
  const f32x2 q = mul2(y, y);
  f32x2 p = fma2(q, both(0.00152817f), both(-0.00729639f));
  p = fma2(q, p, both(0.02121742f));
  p = fma2(q, p, both(-0.05382224f));
  p = fma2(q, p, both(0.13331741f));
  p = fma2(q, p, both(-0.33333272f));
  return fma2(mul2(y, q), p, y);
}
__device__ __forceinline__ float tanh_any(float y) { return fabsf(y) <= TANH_SMALL ? tanh_short(y) : tanhf(y); }
// Caps up to this: two scores differ by 2 cap at most, exp(2 cap) is far inside the range of 32-bit numbers and of bfloat16, and the weights need no
// maximum: their scale is that of a score of zero, or 2^-SCALE_ROOM of the cap's own where that is more, so that sums over many keys stay in
// range.  (At the cap's own scale, far above most scores, an exponent's argument was rounded four times as coarsely.)
constexpr float CAP_AS_SCALE = 38.f, SCALE_ROOM = 32.f;

__global__ void __launch_bounds__(THREADS, HD == 64 ? 2 : 1)
attn_wide_tc_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ Wide a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sq = smem;                                        // [query tile][term][64-wide block][128 rows]
  unsigned char* skv = sq + NX * Q_TILE;                            // [stage][keys | values][64-wide block][BN rows]
  WideBars* bars = reinterpret_cast<WideBars*>(skv + (size_t)STAGES * KV_BYTES);
  const int r = blockIdx.y, g = blockIdx.x, pair = gridDim.z - 1 - blockIdx.z;       // the pairs that see the most keys start first
  const int rep = a.nh / a.nkv, per_tile = BM / rep;               // tokens of a tile
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&bars->kv_full[s]), 1);
      mbar_init(smem_u32(&bars->kv_empty[s]), 1);
    }
    for (int x = 0; x < NX; ++x) {
      for (int b = 0; b < 2; ++b) {
        mbar_init(smem_u32(&bars->s_full[x][b]), 1);
        mbar_init(smem_u32(&bars->p_full[x][b]), 4);
        mbar_init(smem_u32(&bars->pv_done[x][b]), 1);
      }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  pdl_trigger();
  const int t0 = a.row_start[r], q_len = a.row_start[r + 1] - t0, ctx = a.row_ctx[r];
  const bool padding = a.positions != nullptr && q_len > 0 && a.positions[t0] < 0;   // sees no key: its output is zero
  int tok0[NX], n_tok[NX], n_tiles[NX];                    // (constant indices: dynamic ones would put them into memory)
  // the tiles of keys that some row of the pair sees, from the first token's window to each query tile's last token
  const int key_lo = a.window > 0 ? max(0, ctx + NX * pair * per_tile - a.window + 1) : 0, j0 = key_lo / BN;
  int n_all = 0, key_hi = 0;
#pragma unroll
  for (int x = 0; x < NX; ++x) {
    tok0[x] = (NX * pair + x) * per_tile;
    n_tok[x] = ctx >= 0 ? max(0, min(per_tile, q_len - tok0[x])) : 0;
    n_tiles[x] = n_tok[x] > 0 && !padding ? (ctx + tok0[x] + n_tok[x] + BN - 1) / BN - j0 : 0;
    n_all = max(n_all, n_tiles[x]);
    if (n_tok[x] > 0) key_hi = ctx + tok0[x] + n_tok[x];
  }
  // the queries' terms, as the products read them (128-byte swizzle)
  if (n_all > 0) {
    for (int e = threadIdx.x; e < NX * BM * (HD / 8); e += THREADS) {
      const int x = e / (BM * (HD / 8)), row = e / (HD / 8) % BM, c = e % (HD / 8), tok = row / rep;
      uint4 h = make_uint4(0u, 0u, 0u, 0u), l = h;
      if (tok < (x ? n_tok[NX - 1] : n_tok[0])) {
        const float2* p = reinterpret_cast<const float2*>(a.q + (long long)(t0 + (NX * pair + x) * per_tile + tok) * a.q_stride + (long long)(g * rep + row - tok * rep) * HD + c * 8);
        const float2 v0 = p[0], v1 = p[1], v2 = p[2], v3 = p[3];
        two_terms(v0.x, v0.y, h.x, l.x); two_terms(v1.x, v1.y, h.y, l.y);
        two_terms(v2.x, v2.y, h.z, l.z); two_terms(v3.x, v3.y, h.w, l.w);
      }
      unsigned char* at = sq + x * Q_TILE + (c >> 3) * BLOCK + row * 128 + (((c & 7) ^ (row & 7)) << 4);
      *reinterpret_cast<uint4*>(at) = h;
      *reinterpret_cast<uint4*>(at + Q_TERM) = l;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ keys and values: lane p owns page p of a tile
    const int* bt = a.block_tables + (long long)r * a.bt_stride;
    const int pages = BN / a.page_size;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int j = 0; j < n_all; ++j) {
      const uint32_t fb = smem_u32(&bars->kv_full[stage]);
      ok = mbar_wait(smem_u32(&bars->kv_empty[stage]), phase ^ 1);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      if (lane == 0) mbar_expect_tx(fb, KV_BYTES);
      __syncwarp();
      if (lane < pages) {
        unsigned char* sk = skv + (size_t)stage * KV_BYTES;
        const int key0 = (j0 + j) * BN + lane * a.page_size;
        long long krow = a.kv_rows, vrow = a.kv_rows;       // out of bounds: the box reads as zeros
        if (key0 < key_hi && key0 + a.page_size > key_lo) {
          const int blk = key0 / a.page_size, page = blk < a.bt_stride ? bt[blk] : -1;
          if (page < 0 || page >= a.num_pages) {
            fmx_set_status(a.status, FMX_BAD_PAGE, page, r);
          } else {
            krow = (((long long)page * 2 + 0) * a.nkv + g) * a.page_size;
            vrow = (((long long)page * 2 + 1) * a.nkv + g) * a.page_size;
          }
        }
        const int off = lane * a.page_size * 128;
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) {
          tma_load_2d(smem_u32(sk + kb * BN * 128 + off), &map_kv, kb * 64, (int)krow, fb);
          tma_load_2d(smem_u32(sk + KV_HALF + kb * BN * 128 + off), &map_kv, kb * 64, (int)vrow, fb);
        }
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (!ok && lane == 0) fmx_set_status(a.status, FMX_WAIT_EXPIRED, 31, blockIdx.x);
  } else if (warp == 1) {
    // ------------------------------------------------------------------ products: whichever query tile has its inputs goes next
    const bool leader = elect_one();
    const uint32_t idesc_s = make_idesc(BM, BN, 0), idesc_o = make_idesc(BM, HD, 1);
    int qk[NX] = {}, pv[NX] = {}, released = 0;
    bool ok = true;
    long long t_last = clock64();
    while (ok && (pv[0] < n_tiles[0] || pv[NX - 1] < n_tiles[NX - 1])) {
      bool progress = false;
#pragma unroll
      for (int x = 0; x < NX; ++x) {
        const int j = qk[x], st = j % STAGES;
        if (j < n_tiles[x] &&
            __all_sync(0xffffffffu, mbar_test(smem_u32(&bars->kv_full[st]), (uint32_t)((j / STAGES) & 1)) &&
                                        (j < 2 || mbar_test(smem_u32(&bars->pv_done[x][j & 1]), (uint32_t)(((j >> 1) - 1) & 1))))) {
          tc_fence_after();
          const uint32_t q_lo = desc_lo_k128(smem_u32(sq + x * Q_TILE)), k_lo = desc_lo_k128(smem_u32(skv + (size_t)st * KV_BYTES));
          if (leader) {
#pragma unroll
            for (int term = 1; term >= 0; --term)
#pragma unroll
              for (int kb = 0; kb < KB; ++kb)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  umma_f16(tmem + S_COL + (2 * x + (j & 1)) * BN, desc_sw128(q_lo + ((term * Q_TERM + kb * BLOCK) >> 4) + 2 * k),
                           desc_sw128(k_lo + (kb * BN * 128 >> 4) + 2 * k), idesc_s, term == 0 || kb || k ? 1u : 0u);
            umma_commit(smem_u32(&bars->s_full[x][j & 1]));
          }
          __syncwarp();
          ++qk[x];
          progress = true;
        }
        const int i = pv[x], sv = i % STAGES;
        if (i < qk[x] && __all_sync(0xffffffffu, mbar_test(smem_u32(&bars->p_full[x][i & 1]), (uint32_t)((i >> 1) & 1)))) {
          tc_fence_after();
          const uint32_t p_hi = tmem + S_COL + (2 * x + (i & 1)) * BN, p_lo = p_hi + BN / 2;
          const uint32_t v_lo = desc_lo_mn128(smem_u32(skv + (size_t)sv * KV_BYTES + KV_HALF), BN * 128);
          if (leader) {
#pragma unroll
            for (int term = 1; term >= 0; --term)
#pragma unroll
              for (int k = 0; k < BN / 16; ++k)
                umma_f16_ts(tmem + O_COL + x * HD, (term ? p_lo : p_hi) + 8 * k, desc_sw128(v_lo + (k * 16 * 128 >> 4)), idesc_o,
                            i > 0 || term == 0 || k ? 1u : 0u);
            umma_commit(smem_u32(&bars->pv_done[x][i & 1]));
          }
          __syncwarp();
          ++pv[x];
          progress = true;
        }
      }
      while (released < n_all && (released >= n_tiles[0] || pv[0] > released) &&
             (released >= n_tiles[NX - 1] || pv[NX - 1] > released)) {
        if (leader) umma_commit(smem_u32(&bars->kv_empty[released % STAGES]));
        __syncwarp();
        ++released;
      }
      if (progress) t_last = clock64();
      else if (__any_sync(0xffffffffu, clock64() - t_last > WAIT_CYCLES)) ok = false;
    }
    if (!ok && leader) fmx_set_status(a.status, FMX_WAIT_EXPIRED, 32, blockIdx.x);
    // (what was issued is waited for below, before tensor memory is given back: by the softmax groups where all went well)
    if (!ok) {
      if (leader) umma_commit(smem_u32(&bars->kv_empty[0]));
      for (int i = 0; i < 2; ++i) mbar_wait(smem_u32(&bars->kv_empty[0]), (uint32_t)i);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax and output
    const int x = (warp - 2) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int tok = row / rep, head = g * rep + row - tok * rep;
    const int my_tok0 = x ? tok0[NX - 1] : tok0[0], my_tok = x ? n_tok[NX - 1] : n_tok[0], my_tiles = x ? n_tiles[NX - 1] : n_tiles[0];
    const bool valid = tok < my_tok;
    const int pos = ctx + my_tok0 + tok, lim = valid ? pos : -1, lo = valid && a.window > 0 ? max(0, pos - a.window + 1) : 0;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t o_addr = lanes + O_COL + x * HD;
    const bool capped = a.softcap > 0.f;
    const float sl2 = a.scale * LOG2E, cap_l2 = a.softcap * LOG2E, to_y = capped ? a.scale / a.softcap : 0.f;
    // keys that every row of the tile sees: from the last token's window to the first token's position
    const int sure_lo = a.window > 0 ? ctx + my_tok0 + my_tok - a.window : 0, sure_hi = ctx + my_tok0;
    const bool whole = my_tok == per_tile;
    const bool fixed = capped && a.softcap <= CAP_AS_SCALE;
    float m = fixed ? fmaxf(cap_l2 - SCALE_ROOM, 0.f) : -INFINITY;      // the scale in use (of the scores in base 2)
    float l = 0.f;                             // the row's sum at that scale
    bool ok = true;
    for (int j = 0; j < my_tiles; ++j) {
      const int b = j & 1;
      const uint32_t s_addr = lanes + S_COL + (2 * x + b) * BN;
      if (!mbar_wait(smem_u32(&bars->s_full[x][b]), (uint32_t)((j >> 1) & 1))) { ok = false; break; }
      tc_fence_after();
      const int key0 = (j0 + j) * BN;
      const bool below = whole && key0 + BN - 1 <= sure_hi, inside = key0 >= sure_lo;      // every row sees this far down; this far back
      const int hi = lim - key0, back = lo - key0;
      float v[64];
      auto load = [&]() {
        tmem_ld64(s_addr, reinterpret_cast<uint32_t(&)[64]>(v));
        tmem_ld_wait();
      };
      load();
      if (!fixed) {
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (below && inside) {
#pragma unroll
          for (int i = 0; i < 64; i += 2) mx[(i >> 1) & 3] = fmaxf(fmaxf(mx[(i >> 1) & 3], v[i]), v[i + 1]);
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) mx[i & 3] = fmaxf(mx[i & 3], i <= hi && i >= back ? v[i] : -INFINITY);
        }
        float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        top = capped ? (top == -INFINITY ? top : cap_l2 * tanh_any(top * to_y)) : top * sl2;        // scale > 0, the tangent rises: the maximum commutes
        const bool grow = top > m + 8.0f || (m == -INFINITY && top > -INFINITY);
        float alpha = 1.0f;
        if (grow) {
          alpha = exp2_fast(m - top);          // 0 while nothing has been summed
          m = top;
        }
        if (j > 0 && __any_sync(0xffffffffu, grow)) {      // the output so far is brought to the new scale
          if (!mbar_wait(smem_u32(&bars->pv_done[x][b ^ 1]), (uint32_t)(((j - 1) >> 1) & 1))) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < HD; c += 32) {
            uint32_t o[32];
            tmem_ld32(o_addr + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st32(o_addr + c, o);
          }
          l *= alpha;
        }
      }
      const float m_use = m == -INFINITY ? 0.f : m;
      bool large = false;
      if (capped) {
        float ma[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 64; i += 2) ma[(i >> 1) & 3] = fmaxf(fmaxf(ma[(i >> 1) & 3], fabsf(v[i])), fabsf(v[i + 1]));
        large = __any_sync(0xffffffffu, !(fmaxf(fmaxf(ma[0], ma[1]), fmaxf(ma[2], ma[3])) * to_y <= TANH_SMALL));
        if (large) {                           // some score needs the tangent's longer form: all are capped where they lie, in units of the cap
#pragma unroll 1
          for (int i0 = 0; i0 < 64; i0 += 16) {
            uint32_t u[16];
            float t[16];
            tmem_ld16(s_addr + i0, u);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) t[i] = tanh_any(__uint_as_float(u[i]) * to_y);
            tmem_st16(s_addr + i0, t);
            tmem_st_wait();
          }
          load();
        }
      }
      const float by = capped ? cap_l2 : sl2;
      f32x2 sum[4] = {0ull, 0ull, 0ull, 0ull};
      uint32_t first[32], rest[32];
      // one loop for each form that a tile can take: a branch inside would hold every score up
      auto weights = [&](auto tangent, auto masked) {
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          float p[2];
          f32x2 t = pair_of(v[i], v[i + 1]);
          if (decltype(tangent)::value) t = tanh_short(mul2(t, pair_of(to_y, to_y)));
          halves(fma2(t, pair_of(by, by), pair_of(-m_use, -m_use)), p[0], p[1]);
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            p[n] = exp2_fast(p[n]);
            if (decltype(masked)::value) p[n] = i + n <= hi && i + n >= back ? p[n] : 0.f;
          }
          const f32x2 both = pair_of(p[0], p[1]);
          sum[(i >> 1) & 3] = add2(sum[(i >> 1) & 3], both);
          const unsigned h = pack2(p[0], p[1]);
          float r0, r1;
          halves(sub2(both, pair_of(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u))), r0, r1);
          first[i >> 1] = h;
          rest[i >> 1] = pack2(r0, r1);
        }
      };
      if (capped && !large) {
        if (below && inside) weights(std::true_type{}, std::false_type{});
        else weights(std::true_type{}, std::true_type{});
      } else {
        if (below && inside) weights(std::false_type{}, std::false_type{});
        else weights(std::false_type{}, std::true_type{});
      }
      tmem_st32(s_addr, first);                // over the tile's own scores
      tmem_st32(s_addr + BN / 2, rest);
      tmem_st_wait();
      l += pair_sum(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])));
      // keys out of sight share pages with others: their values must be zeros, since 0 times an infinity would poison the product (both
      // groups write the same zeros)
      if (key0 + BN > key_hi || key0 < key_lo) {
        const int st = j % STAGES;
        if (!mbar_wait(smem_u32(&bars->kv_full[st]), (uint32_t)((j / STAGES) & 1))) { ok = false; break; }
        if (row < BN && (key0 + row >= key_hi || key0 + row < key_lo)) {
          unsigned char* sv = skv + (size_t)st * KV_BYTES + KV_HALF + row * 128;
#pragma unroll
          for (int kb = 0; kb < KB; ++kb)
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) *reinterpret_cast<uint4*>(sv + kb * BN * 128 + ch * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars->p_full[x][b]));
    }
    if (ok && my_tiles > 0) ok = mbar_wait(smem_u32(&bars->pv_done[x][(my_tiles - 1) & 1]), (uint32_t)(((my_tiles - 1) >> 1) & 1));
    if (!ok) {
      if (lane == 0) fmx_set_status(a.status, FMX_WAIT_EXPIRED, 33, blockIdx.x);
    } else if (my_tok > 0) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      bf16* op = a.out + (long long)(t0 + my_tok0 + tok) * a.out_stride + (long long)head * HD;
#pragma unroll
      for (int c = 0; c < HD; c += 32) {
        uint32_t v[32];
        if (my_tiles > 0) {
          tmem_ld32(o_addr + c, v);            // the whole warp loads; valid rows store
          tmem_ld_wait();
        }
        if (valid) {
          unsigned w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = my_tiles > 0 ? pack2(__uint_as_float(v[2 * i]) * inv, __uint_as_float(v[2 * i + 1]) * inv) : 0u;
          if (a.out16) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(op + c + 2 * i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) *reinterpret_cast<unsigned*>(op + c + 2 * i) = w[i];
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}
}  // namespace

// As fmx_attn_prefill_wide_masked without kept tokens, runs of positions, shares and terms without a value, over pages of keys and values,
// for up to 16 query heads per kv head, a page size of at least 8 that divides the 64 keys of a tile
// and a positive scale.
FMX_EXPORT int fmx_attn_wide_tc(const float* q, long long q_stride, const void* kv, const int* block_tables, int bt_stride,
                                const int* row_start, const int* row_ctx, const int* positions, void* out, long long out_stride, int rows,
                                int max_q_len, int nh, int nkv, int page_size, long long num_pages, float scale, float softcap, int window,
                                int* status, cudaStream_t stream) {
  if (rows == 0 || max_q_len == 0) return 0;
  if (rows < 0 || nh <= 0 || nkv <= 0 || nh % nkv || nh / nkv > 16 || window < 0 || !(scale > 0.f))
    return fmx_fail("fmx_attn_wide_tc: bad sizes rows=%d nh=%d nkv=%d window=%d scale=%g", rows, nh, nkv, window, scale);
  if (page_size < 8 || BN % page_size) return fmx_fail("fmx_attn_wide_tc: a page of %d tokens does not tile %d keys", page_size, BN);
  if (q_stride % 2 || ((uintptr_t)q & 7) || out_stride % 2 || ((uintptr_t)out & 3) || out_stride < (long long)nh * HD || ((uintptr_t)kv & 15))
    return fmx_fail("fmx_attn_wide_tc: queries in 8-byte pairs, outputs in 4-byte pairs, rows at least nh*hd wide, pages on 16 bytes");
  const int rep = nh / nkv, per_pair = NX * (BM / rep);
  const long long pairs = ((long long)max_q_len + per_pair - 1) / per_pair, kv_rows = num_pages * 2 * nkv * page_size;
  if (rows > 65535 || pairs > 65535) return fmx_fail("fmx_attn_wide_tc: too many rows or query tokens for one launch");
  if (kv_rows >= 2147483647LL) return fmx_fail("fmx_attn_wide_tc: the cache has too many rows for a 32-bit coordinate");
  EncodeTiledFn enc = encode_fn();
  if (enc == nullptr) return fmx_fail("fmx_attn_wide_tc: cuTensorMapEncodeTiled is not available from this driver");
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)HD, (cuuint64_t)kv_rows};
  const cuuint64_t strides[1] = {(cuuint64_t)HD * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)page_size}, estr[2] = {1, 1};
  const CUresult rc = enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(kv), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return fmx_fail("fmx_attn_wide_tc: encoding the cache map failed with code %d", (int)rc);
  static thread_local int raised = -1;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess && device != raised) {
    e = cudaFuncSetAttribute(attn_wide_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e == cudaSuccess) raised = device;
  }
  if (e != cudaSuccess) return fmx_fail("fmx_attn_wide_tc: %zu bytes of shared memory refused: %s", SMEM, cudaGetErrorString(e));
  const Wide a = {q, q_stride, block_tables, row_start, row_ctx, positions, (bf16*)out, out_stride, num_pages, kv_rows, bt_stride, nh, nkv, page_size,
                  window, scale, softcap, out_stride % 8 == 0 && ((uintptr_t)out & 15) == 0 ? 1 : 0, status};
  e = fmx_launch(attn_wide_tc_kernel, dim3(nkv, rows, (unsigned)pairs), dim3(THREADS), SMEM, stream, map, a);
  if (e != cudaSuccess) return fmx_fail("fmx_attn_wide_tc: launch failed: %s", cudaGetErrorString(e));
  return 0;
}
#else
#include "common.cuh"
FMX_EXPORT int fmx_attn_wide_tc(const float*, long long, const void*, const int*, int, const int*, const int*, const int*, void*, long long, int, int, int,
                                int, int, long long, float, float, int, int*, cudaStream_t) {
  return fmx_fail("fmx_attn_wide_tc: this head size has no tensor-memory attention kernel");
}
#endif
