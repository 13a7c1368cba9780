// C[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) with 32-bit activations A and a matrix W whose values are bfloat16, to 32-bit accuracy
// on the fifth-generation tensor cores: an activation goes in as three bfloat16 terms (three_terms.cuh) that hold all its 24 bits,
// a weight as itself, so that no product is rounded at all.
//
// One order of sums for every M.  The tensor cores cut their sums off instead of rounding them, so they add up 64 k only:
// the small terms first, then the leading ones (four sums of the full size).  Such blocks of 64 k are added up in rounded
// 32-bit sums in registers, k ascending, over `splits` shares of K, and the shares' sums one after the other.  The
// shares follow from the matrix's N and K alone (plan_splits; a product over some of a matrix's rows takes the whole matrix's)
// and a product's column does not depend on the other columns, so a token's result is the same whichever other tokens share the
// step, and whichever other features the product.
//
//   split       lays the activations' terms out in memory, three matrices one under the other.
//   warp 0      brings blocks of W (128 features x 64 k) and of the terms (up to 128 tokens x 64 k each) by TMA.
//   warp 1      issues the products: W's features are the 128 rows, the tokens the columns, twelve a block.
//   warps 2-9   add a block's sums up: a warp owns 32 features and every other 16 tokens.
//
// Where the tiles fill the GPU a CTA walks all of K (the shares' sum waits in tensor memory); else the shares of a tile go to
// the CTAs of a cluster, which add them up in order through one another's shared memory.
//
// Bound by the products and the clock that they leave under the power limit (2,048 tokens: 1.24 PFLOP/s of bfloat16, three products to a
// 32-bit one), below some 64 tokens by twelve products of at least 44 clocks a block.  Against 32-bit multiply-adds over the widened
// matrix (gemm_simple.cu), the split with it, weights from memory, us: 16,384 x 2,048, 1 token 29 -> 19, 333 592 -> 65, 1,024 1,314 -> 168;
// 2,048 x 8,192 55 -> 14, 474 -> 60, 841 -> 101.  Error against 64-bit, of the result's norm: 1.2e-7 to 1.6e-7, multiply-adds 0.8e-6 to 2.1e-6.
#include "common.cuh"
#include "tcgen05.cuh"
#include "three_terms.cuh"

namespace {
using namespace fmx_tc;
constexpr int TF = 128, BK = 64, MAX_TOKENS = 128, MAX_SPLITS = 8, MAX_STAGES = 8;
constexpr int EPI_WARPS = 8, THREADS = 32 * (2 + EPI_WARPS);
constexpr int W_BYTES = TF * BK * 2;
constexpr int TMEM_COLS = 512, SUM_COL = 256;              // two buffers of a block's sums, and the sum over the shares so far
constexpr int APART = 8;
constexpr size_t SMEM_MAX = 227 * 1024, SMEM_EXTRA = 1024 /* alignment */ + 256 /* barriers */;
static_assert(MAX_TOKENS * TF * 4 <= 3 * (W_BYTES + 3 * MAX_TOKENS * BK * 2), "a share's sums fit where the blocks were");
static_assert((2 * MAX_STAGES + 5) * 8 + 4 <= 256, "the barriers outgrow their corner of shared memory");

struct Three {
  const float* bias;
  float* C;
  long long ldc;
  int M, N, K, tokens, tiles_t, tiles, stages, splits, shares_apart;        // tokens: of a tile; shares_apart: a cluster takes a tile's shares
  int c16;                                                 // rows of C start on 16 bytes
  int* status;
};

__device__ __forceinline__ int share_start(int s, int blocks, int splits) { return s * blocks / splits; }

__global__ void __launch_bounds__(THREADS, 1)
gemm_three_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ Three a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int plane = a.tokens * BK * 2, stage_bytes = W_BYTES + 3 * plane;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)a.stages * stage_bytes);
  uint64_t *full = bars, *empty = bars + MAX_STAGES, *acc_full = bars + 2 * MAX_STAGES, *acc_empty = acc_full + 2, *drain = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int blocks = (a.K + BK - 1) / BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&acc_full[i]), 1);
      mbar_init(smem_u32(&acc_empty[i]), EPI_WARPS);
    }
    mbar_init(smem_u32(drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // this CTA's tiles, and its blocks of each: all of K, or one share of it
  const int share = a.shares_apart ? (int)blockIdx.x % a.splits : 0;
  const int first = a.shares_apart ? (int)blockIdx.x / a.splits : (int)blockIdx.x;
  const int step = a.shares_apart ? a.tiles : (int)gridDim.x;               // (shares apart: one tile a cluster)
  const int b_lo = a.shares_apart ? share_start(share, blocks, a.splits) : 0;
  const int b_hi = a.shares_apart ? share_start(share + 1, blocks, a.splits) : blocks;
  const int m_first = first % a.tiles_t * a.tokens, n_first = first / a.tiles_t * TF;
  const int mine = first < a.tiles ? ((a.tiles - 1 - first) / step + 1) * (b_hi - b_lo) : 0;       // this CTA's blocks
  bool ok = true;

  if (warp == 0) {                               // ---- blocks of W and of the terms
    const bool leader = elect_one();
    int stage = 0, t = first, b = b_lo, m0 = m_first, n0 = n_first;
    uint32_t phase = 0;
    // weights are nothing that a kernel before this one writes: the first blocks of W are on their way before the terms are waited for
    const int ahead = min(a.stages, mine);
    if (leader)
      for (int i = 0, ti = first, bi = b_lo; i < ahead; ++i) {
        const uint32_t fb = smem_u32(&full[i]);
        mbar_expect_tx(fb, (uint32_t)stage_bytes);
        tma_load_2d(smem_u32(smem + (size_t)i * stage_bytes), &map_w, bi * BK, ti / a.tiles_t * TF, fb);
        if (++bi == b_hi) { bi = b_lo; ti += step; }
      }
    __syncwarp();
    pdl_wait();
    for (int i = 0; i < mine; ++i) {
      if (i >= ahead && !mbar_wait(smem_u32(&empty[stage]), phase ^ 1)) { ok = false; break; }
      if (leader) {
        const uint32_t fb = smem_u32(&full[stage]), dst = smem_u32(smem + (size_t)stage * stage_bytes);
        if (i >= ahead) {
          mbar_expect_tx(fb, (uint32_t)stage_bytes);
          tma_load_2d(dst, &map_w, b * BK, n0, fb);
        }
#pragma unroll
        for (int term = 0; term < 3; ++term) tma_load_2d(dst + W_BYTES + term * plane, &map_x, b * BK, term * a.M + m0, fb);
      }
      if (++stage == a.stages) { stage = 0; phase ^= 1; }
      if (++b == b_hi) {
        b = b_lo;
        t += step;
        m0 = t % a.tiles_t * a.tokens;
        n0 = t / a.tiles_t * TF;
      }
    }
    if (!ok && leader) {
      fmx_set_status(a.status, FMX_WAIT_EXPIRED, 1, blockIdx.x);
      for (int s = 0; s < ahead; ++s) mbar_wait(smem_u32(&full[s]), 0) || mbar_wait(smem_u32(&full[s]), 1);      // its own copies in flight land first
    }
    __syncwarp();
  } else if (warp == 1) {                        // ---- products
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc(TF, a.tokens), plane16 = (uint32_t)plane >> 4;
    const uint32_t base = desc_lo_k128(smem_u32(smem));
    int stage = 0, buf = 0;
    uint32_t phase = 0, acc_phase = 0;
    ok = mine == 0 || mbar_wait(smem_u32(&full[0]), 0);
    for (int i = 0; i < mine && ok; ++i) {
      tc_fence_after();
      const uint32_t sw = base + stage * (stage_bytes >> 4), sx = sw + (W_BYTES >> 4), d = tmem + (uint32_t)(buf * MAX_TOKENS);
      auto products = [&](int term) {
        if (leader)
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_f16(d, desc_sw128(sw + 2 * k), desc_sw128(sx + term * plane16 + 2 * k), idesc, term < 2 || k > 0 ? 1u : 0u);
      };
      products(2);
      products(1);
      // is the next block there?  Asked while this block's products run: behind them the two waits are time the tensor pipe stands still
      const int old = stage, old_buf = buf;
      if (++stage == a.stages) { stage = 0; phase ^= 1; }
      if (++buf == 2) { buf = 0; acc_phase ^= 1; }
      const bool there = i + 1 < mine && mbar_test(smem_u32(&acc_empty[buf]), acc_phase ^ 1) && mbar_test(smem_u32(&full[stage]), phase);
      products(0);
      if (leader) {
        umma_commit(smem_u32(&empty[old]));
        umma_commit(smem_u32(&acc_full[old_buf]));
      }
      __syncwarp();
      if (i + 1 < mine && !__all_sync(0xffffffffu, there))
        ok = mbar_wait(smem_u32(&acc_empty[buf]), acc_phase ^ 1) && mbar_wait(smem_u32(&full[stage]), phase);
    }
    if (!ok && leader) {
      fmx_set_status(a.status, FMX_WAIT_EXPIRED, 2, blockIdx.x);
      umma_commit(smem_u32(drain));              // what was issued may still run: tensor memory is not freed under it
      mbar_wait(smem_u32(drain), 0);
    }
    __syncwarp();
  } else {                                       // ---- sums over K
    pdl_wait();
    pdl_trigger();
    const int quarter = warp & 3, half = (warp - 2) >> 2, chunks = a.tokens / 16;       // this warp: chunks half, half + 2, ...
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    int buf = 0;
    uint32_t acc_phase = 0;
    for (int t = first; t < a.tiles && ok; t += step) {
      const int m0 = t % a.tiles_t * a.tokens, n = t / a.tiles_t * TF + quarter * 32 + lane;
      float sum[4][16];
      int s = share, s_lo = b_lo, s_hi = share_start(share + 1, blocks, a.splits);
      for (int b = b_lo; b < b_hi; ++b) {
        if (!mbar_wait(smem_u32(&acc_full[buf]), acc_phase)) { ok = false; break; }
        tc_fence_after();
        const bool fresh = b == s_lo;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (2 * i + half < chunks) {
            uint32_t v[16];
            tmem_ld16(lanes + buf * MAX_TOKENS + (2 * i + half) * 16, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) sum[i][e] = fresh ? __uint_as_float(v[e]) : sum[i][e] + __uint_as_float(v[e]);
          }
        tc_fence_before();
        __syncwarp();                            // one arrival a warp: those of a whole warp queue up behind one another
        if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));
        if (++buf == 2) { buf = 0; acc_phase ^= 1; }
        if (b + 1 == s_hi) {
          if (!a.shares_apart && a.splits > 1) {            // the sum over the shares: in tensor memory, but for the last one
            const bool last = s + 1 == a.splits;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (2 * i + half >= chunks) continue;
              const uint32_t at = lanes + SUM_COL + (2 * i + half) * 16;
              uint32_t v[16];
              if (s > 0) {
                tmem_ld16(at, v);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e) sum[i][e] = __uint_as_float(v[e]) + sum[i][e];
              }
              if (!last) tmem_st16(at, sum[i]);
            }
            if (!last) tmem_st_wait();
          }
          s_lo = s_hi;
          s_hi = share_start(++s + 1, blocks, a.splits);
        }
      }
      if (!ok) break;
      if (a.shares_apart) {                      // the ring is read through: this share's sums take its place, [token][feature]
        float* mine = reinterpret_cast<float*>(smem);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (2 * i + half < chunks)
#pragma unroll
            for (int e = 0; e < 16; ++e) mine[((2 * i + half) * 16 + e) * TF + quarter * 32 + lane] = sum[i][e];
      } else if (n < a.N) {
        const float bias = a.bias != nullptr ? a.bias[n] : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (2 * i + half < chunks)
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const int m = m0 + (2 * i + half) * 16 + e;
              if (m < a.M) a.C[(long long)m * a.ldc + n] = a.bias != nullptr ? sum[i][e] + bias : sum[i][e];
            }
      }
    }
    if (!ok && lane == 0) fmx_set_status(a.status, FMX_WAIT_EXPIRED, 3, blockIdx.x);
  }

  if (a.shares_apart) {                          // uniform over the grid: every thread of a cluster meets here, whatever its waits did
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int valid = min(a.tokens, a.M - m_first) * (TF / 4);
    for (int e = share * (int)blockDim.x + (int)threadIdx.x; e < valid; e += a.splits * (int)blockDim.x) {
      const uint32_t at = smem_u32(smem) + e * 16;
      float4 v[MAX_SPLITS];
#pragma unroll
      for (int s = 0; s < MAX_SPLITS; ++s)
        if (s < a.splits) {
          uint32_t peer;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(s));
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v[s].x), "=f"(v[s].y), "=f"(v[s].z), "=f"(v[s].w) : "r"(peer) : "memory");
        }
      float4 sum = v[0];
#pragma unroll
      for (int s = 1; s < MAX_SPLITS; ++s)
        if (s < a.splits) { sum.x += v[s].x; sum.y += v[s].y; sum.z += v[s].z; sum.w += v[s].w; }
      const int n = n_first + e % (TF / 4) * 4;
      const float r[4] = {sum.x, sum.y, sum.z, sum.w};
      float* c = a.C + (long long)(m_first + e / (TF / 4)) * a.ldc + n;
      if (a.bias == nullptr && a.c16 && n + 4 <= a.N) {
        *reinterpret_cast<float4*>(c) = sum;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < a.N) c[j] = a.bias != nullptr ? r[j] + a.bias[n + j] : r[j];
      }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");      // a peer may still read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// Shares of K: of N and K alone, for a B200's 148 SMs, of which clusters of s CTAs reach AT_ONCE[s - 1] x s.  With the blocks of K that the
// busiest SM takes at few tokens and two more a share for adding them up, the fewest: 2,048 x 8,192, one token: 6 shares 13 us, 8
// (two rounds of clusters) 20, 4 17.
int plan_splits(int N, int K) {
  static const int AT_ONCE[MAX_SPLITS] = {148, 74, 45, 33, 26, 22, 15, 15};
  const int tiles = (N + TF - 1) / TF, blocks = (K + BK - 1) / BK;
  int best = 1;
  long long least = -1;
  for (int s = 1; s <= MAX_SPLITS && s <= blocks; ++s) {
    const long long cost = (long long)((tiles + AT_ONCE[s - 1] - 1) / AT_ONCE[s - 1]) * ((blocks + s - 1) / s) + 2 * s;
    if (least < 0 || cost < least) { least = cost; best = s; }
  }
  return best;
}

// eight values -> eight bfloat16 of each of their three terms
__device__ __forceinline__ void terms_of(const float (&v)[8], uint4 (&t)[3]) {
  float most = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) most = fmaxf(most, fabsf(v[j]));
  if (most < 3.3e38f) {                          // below what rounds to an infinity in bfloat16
    three_terms(v[0], v[1], t[0].x, t[1].x, t[2].x); three_terms(v[2], v[3], t[0].y, t[1].y, t[2].y);
    three_terms(v[4], v[5], t[0].z, t[1].z, t[2].z); three_terms(v[6], v[7], t[0].w, t[1].w, t[2].w);
  } else {
    three_terms_large(v[0], v[1], t[0].x, t[1].x, t[2].x); three_terms_large(v[2], v[3], t[0].y, t[1].y, t[2].y);
    three_terms_large(v[4], v[5], t[0].z, t[1].z, t[2].z); three_terms_large(v[6], v[7], t[0].w, t[1].w, t[2].w);
  }
}

// The activations' three terms, one [M, K] matrix under the other.
__global__ void __launch_bounds__(256)
split_kernel(const float* x, long long ldx, bf16* out, int M, int K, int x16) {
  pdl_wait();
  pdl_trigger();
  const int per_row = K / 8;
  const long long all = (long long)M * per_row;
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < all; e += (long long)gridDim.x * 256) {
    const long long m = e / per_row;
    const int k = (int)(e - m * per_row) * 8;
    const float* p = x + m * ldx + k;
    float v[8];
    if (x16) {
      const float4 u = *reinterpret_cast<const float4*>(p), w = *reinterpret_cast<const float4*>(p + 4);
      v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w; v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = p[j];
    }
    uint4 t[3];
    terms_of(v, t);
#pragma unroll
    for (int term = 0; term < 3; ++term) *reinterpret_cast<uint4*>(out + ((long long)term * M + m) * K + k) = t[term];
  }
}

// Results that are not finite, worked out again from the operands themselves in one 32-bit sum: an infinite weight meets an activation's
// smaller terms, zeros or of the other sign, and makes a NaN of what is an infinity.  (Inside the product, where no weight is infinite
// as a rule, looking for them costs 1 to 4 %.)
__global__ void __launch_bounds__(256)
not_finite_kernel(const float* x, long long ldx, const bf16* w, long long ldw, const float* bias, float* C, long long ldc, int M, int N, int K) {
  pdl_wait();
  pdl_trigger();
  const long long all = (long long)M * N;
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < all; e += (long long)gridDim.x * 256) {
    const long long m = e / N, n = e - m * N;
    if (isfinite(C[m * ldc + n])) continue;
    float s = 0.f;
    for (int k = 0; k < K; ++k) s = fmaf(x[m * ldx + k], __bfloat162float(w[n * ldw + k]), s);
    C[m * ldc + n] = bias != nullptr ? s + bias[n] : s;
  }
}

}  // namespace

// After fmx_gemm_three, over a matrix that nobody has looked through for infinities: see not_finite_kernel.
FMX_EXPORT int fmx_gemm_three_not_finite(const float* A, long long lda, const void* W, long long ldw, const float* bias, float* C, long long ldc,
                                         int M, int N, int K, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  const long long want = ((long long)M * N + 255) / 256, most = 16LL * fmx_num_sms();
  const cudaError_t e = fmx_launch(not_finite_kernel, dim3((unsigned)(want < most ? want : most)), dim3(256), 0, stream, A, lda, (const bf16*)W, ldw,
                                   bias, C, ldc, M, N, K);
  return e == cudaSuccess ? 0 : fmx_fail("fmx_gemm_three_not_finite: launch failed: %s", cudaGetErrorString(e));
}

// Into how many shares a product of N features over K is split, whatever its number of tokens.
FMX_EXPORT int fmx_gemm_three_splits(int N, int K) { return N > 0 && K > 0 ? plan_splits(N, K) : 0; }

// Tokens whose terms the workspace holds at most, 256 MB of them (whole tiles, and one at least): a product of more goes in waves of so
// many, whose results are the same bits.  Sizes with more than one wave (5,376 tokens over 8,192) fill the GPU many times over.
FMX_EXPORT int fmx_gemm_three_rows(int K) {
  const long long rows = K > 0 ? (256LL << 20) / (6LL * K) / MAX_TOKENS * MAX_TOKENS : 0;
  return rows < MAX_TOKENS ? MAX_TOKENS : (int)rows;
}

// Bytes of workspace that a product of M tokens over K takes: the three terms of a wave's activations.
FMX_EXPORT long long fmx_gemm_three_bytes(int M, int K) {
  const int rows = fmx_gemm_three_rows(K);
  return 6LL * (M < rows ? M : rows) * K;
}

namespace {
int run_wave(const float* A, long long lda, const void* W, long long ldw, const float* bias, float* C, long long ldc, int M, int N, int K,
             int whole_n, void* ws, int sms, int* status, cudaStream_t stream) {
  Three a = {};
  a.bias = bias; a.C = C; a.ldc = ldc; a.M = M; a.N = N; a.K = K; a.status = status;
  a.tiles_t = (M + MAX_TOKENS - 1) / MAX_TOKENS;
  a.tokens = ((M + a.tiles_t - 1) / a.tiles_t + 15) / 16 * 16;
  a.tiles_t = (M + a.tokens - 1) / a.tokens;
  const long long tiles = (long long)a.tiles_t * ((N + TF - 1) / TF);
  if (tiles > 0x7fffffffLL / MAX_SPLITS) return fmx_fail("fmx_gemm_three: M=%d N=%d are too large", M, N);
  a.tiles = (int)tiles;
  a.splits = plan_splits(whole_n, K);
  // A CTA's whole walk over K, or a cluster's shares of it: blocks of K that the busiest SM takes, with APART more for each CTA of a
  // cluster (its start, the ring's filling, the sum over the shares).
  const int blocks = (K + BK - 1) / BK;
  const long long whole = (tiles + sms - 1) / sms * blocks, apart = (tiles * a.splits + sms - 1) / sms * ((blocks + a.splits - 1) / a.splits + APART);
  a.shares_apart = a.splits > 1 && apart < whole ? 1 : 0;
  a.c16 = ldc % 4 == 0 && ((uintptr_t)C & 15) == 0;
  const int stage = W_BYTES + 3 * a.tokens * BK * 2, fit = (int)((SMEM_MAX - SMEM_EXTRA) / stage);
  a.stages = fit < MAX_STAGES ? fit : MAX_STAGES;
  const size_t smem = (size_t)a.stages * stage + SMEM_EXTRA;
  CUtensorMap map_w, map_x;
  if (make_map_k128(&map_w, W, N, K, ldw, TF) || make_map_k128(&map_x, ws, 3LL * M, K, K, a.tokens)) return 1;
  static thread_local int raised = -1;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess && device != raised) {
    e = cudaFuncSetAttribute(gemm_three_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
    if (e == cudaSuccess) raised = device;
  }
  if (e != cudaSuccess) return fmx_fail("fmx_gemm_three: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
  const long long want = ((long long)M * (K / 8) + 255) / 256, most = 8LL * sms;
  e = fmx_launch(split_kernel, dim3((unsigned)(want < most ? want : most)), dim3(256), 0, stream, A, lda, (bf16*)ws, M, K,
                 lda % 4 == 0 && ((uintptr_t)A & 15) == 0 ? 1 : 0);
  if (e != cudaSuccess) return fmx_fail("fmx_gemm_three: launch of the split failed: %s", cudaGetErrorString(e));
  if (a.shares_apart)
    e = fmx_launch_cluster(gemm_three_kernel, dim3(a.tiles * a.splits), dim3(THREADS), smem, stream, dim3(a.splits), map_w, map_x, a);
  else
    e = fmx_launch(gemm_three_kernel, dim3(a.tiles < sms ? a.tiles : sms), dim3(THREADS), smem, stream, map_w, map_x, a);
  if (e != cudaSuccess) return fmx_fail("fmx_gemm_three: launch failed: %s", cudaGetErrorString(e));
  return 0;
}
}  // namespace

// A 32-bit [M, K], W bfloat16 [N, K] with K-contiguous rows that start on 16 bytes, C 32-bit [M, N].  whole_n: features of the matrix
// that W's rows are a part of, whose shares of K the product takes; N where W is all of it.  ws: fmx_gemm_three_bytes on 16
// bytes.  status: the engine's status word (a wait that expires leaves FMX_WAIT_EXPIRED there).
FMX_EXPORT int fmx_gemm_three(const float* A, long long lda, const void* W, long long ldw, const float* bias, float* C, long long ldc,
                              int M, int N, int K, int whole_n, void* ws, int sms, int* status, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  if (M < 0 || N < 0 || K <= 0 || whole_n < N) return fmx_fail("fmx_gemm_three: bad sizes M=%d N=%d of %d K=%d", M, N, whole_n, K);
  if (K % 8 || ldw % 8 || ((uintptr_t)W & 15)) return fmx_fail("fmx_gemm_three: W's rows must start on 16 bytes (K=%d ldw=%lld)", K, ldw);
  if (ws == nullptr || ((uintptr_t)ws & 15)) return fmx_fail("fmx_gemm_three: the workspace is missing or does not lie on 16 bytes");
  if (sms <= 0) sms = fmx_num_sms();
  const int rows = fmx_gemm_three_rows(K);
  for (int m = 0; m < M; m += rows) {
    const int rc = run_wave(A + m * lda, lda, W, ldw, bias, C + m * ldc, ldc, M - m < rows ? M - m : rows, N, K, whole_n, ws, sms, status, stream);
    if (rc != 0) return rc;
    if (M - m <= rows) break;
  }
  return 0;
}
