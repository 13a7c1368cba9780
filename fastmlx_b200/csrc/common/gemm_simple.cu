// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) with 32-bit accumulation in a fixed order.
//
// This is the matrix product of the true 32-bit path and the fallback for mixed element
// types.  Every output element sums its K products one after the other, k ascending, with
// fused multiply-adds; the order does not depend on M, N or the tile an element falls in,
// so a token's result is the same whichever other tokens share the step.
//
// Three kernels with that one order:
//   gemm_nt_tile   32-bit operands in 16-byte rows, more than 20 rows of A: register tiles of 8 x 8, 8 x 4 or 4 x 4 outputs.
//   gemm_nt_few    the same operands, at most 32 rows (decode steps): W streams once, a lane per output feature.
//   gemm_nt_kernel mixed element types and unaligned rows.
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, THREADS = 256;

// Two fused multiply-adds, each rounded as fmaf rounds: (d.x, d.y) += (a.x b.x, a.y b.y).
__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b) {
  unsigned long long& dd = reinterpret_cast<unsigned long long&>(d);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(dd) : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}

__device__ __forceinline__ void copy16(void* dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0));
}

// Bound by the CUDA cores' multiply-adds (an output's sum is one chain in k, so K is never split).
// A block owns TBM x TBN outputs, a thread TM x TN of them: per k it reads TM + TN floats of shared memory in 16-byte
// loads for TM TN multiply-adds (gemm_nt_kernel's scalar loads for 4 x 4 make it wait for shared memory), and issues
// them in pairs of rows.  The next slice of k is on its way from memory in registers while the current one is multiplied.
// 333 x 16,384 x 2,048 and 333 x 2,048 x 8,192 together: 2,127 us with gemm_nt_kernel, 1,073 us here
// (42 % of the CUDA cores' 74.4 TFLOP/s; 2,048 rows of 16,384 x 2,048: 5,980 and 2,620 us, 71 %).
template <int TBM, int TBN, int TM, int TN, int KS>
__global__ void __launch_bounds__((TBM / TM) * (TBN / TN))
gemm_nt_tile(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
             int M, int N, int K, long long lda, long long ldw, long long ldc) {
  constexpr int NT = (TBM / TM) * (TBN / TN);
  constexpr int LA = TBM * KS / 4 / NT, LW = TBN * KS / 4 / NT;       // 16-byte pieces of a slice per thread
  static_assert(LA * NT * 4 == TBM * KS && LW * NT * 4 == TBN * KS, "a slice is shared out evenly");
  __shared__ __align__(16) float As[2][KS][TBM + 4];
  __shared__ __align__(16) float Ws[2][KS][TBN + 4];
  const int tid = threadIdx.x;
  constexpr int TX = TBN / TN;
  const int ty = tid / TX, tx = tid % TX;
  const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
  float4 ra[LA], rw[LW];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int e = tid + i * NT, m = m0 + e / (KS / 4), k = k0 + e % (KS / 4) * 4;
      ra[i] = m < M && k < K ? *reinterpret_cast<const float4*>(A + (long long)m * lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int e = tid + i * NT, n = n0 + e / (KS / 4), k = k0 + e % (KS / 4) * 4;
      rw[i] = n < N && k < K ? *reinterpret_cast<const float4*>(W + (long long)n * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto put = [&](int b) {                          // k-major, so that a thread's rows lie side by side
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int e = tid + i * NT, r = e / (KS / 4), c = e % (KS / 4) * 4;
      As[b][c][r] = ra[i].x; As[b][c + 1][r] = ra[i].y; As[b][c + 2][r] = ra[i].z; As[b][c + 3][r] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int e = tid + i * NT, r = e / (KS / 4), c = e % (KS / 4) * 4;
      Ws[b][c][r] = rw[i].x; Ws[b][c + 1][r] = rw[i].y; Ws[b][c + 2][r] = rw[i].z; Ws[b][c + 3][r] = rw[i].w;
    }
  };
  float2 acc[TM / 2][TN];                          // pairs of rows: one multiplier per column is doubled up, not one per row
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
  const int slices = (K + KS - 1) / KS;
  fetch(0);
  put(0);
  __syncthreads();
  for (int s = 0; s < slices; ++s) {
    const int b = s & 1;
    if (s + 1 < slices) fetch((s + 1) * KS);
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      // a thread's rows and columns come in runs of four, a quarter-warp's runs side by side: no bank is asked twice
      float2 a[TM / 2];
      float w[TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&As[b][kk][i / 4 * (TBM / (TM / 4)) + ty * 4]);
        a[i / 2] = make_float2(v.x, v.y);
        a[i / 2 + 1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&Ws[b][kk][j / 4 * (TBN / (TN / 4)) + tx * 4]);
        w[j] = v.x; w[j + 1] = v.y; w[j + 2] = v.z; w[j + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a[i], make_float2(w[j], w[j]));
    }
    if (s + 1 < slices) {
      put(b ^ 1);                                  // the other buffer was last read before the barrier of the slice before
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + i / 4 * (TBM / (TM / 4)) + ty * 4 + i % 4;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + j / 4 * (TBN / (TN / 4)) + tx * 4 + j % 4;
      if (n >= N) continue;
      float v = i & 1 ? acc[i / 2][j].y : acc[i / 2][j].x;
      if (bias) v += bias[n];
      C[(long long)m * ldc + n] = v;
    }
  }
}

// At most 32 rows: bound by the stream of W, which every block reads once for its FN features, and by the one chain of K
// multiply-adds per output.  Lanes are features (with FN = 16 the half-warps take different rows of A), a lane sums FR
// rows of A for its feature; slices of FK k of W and A come through a ring of cp.async stages.  Products of few features
// (less than 32 per SM) take FN = 16, so that most SMs have a block.
// One row: 16,384 x 2,048 297 us with gemm_nt_kernel, 31 us here; 2,048 x 8,192 582 and 56 us.
// A stage's rows are FK + 4 floats apart, so that eight lanes' 16-byte loads meet no bank twice.  The last four warps copy and
// do nothing else: a multiplying warp's chain of sums does not wait for address arithmetic.
constexpr int COPY_WARPS = 4;

template <int FN, int FR, int STAGES, int FK>
__global__ void __launch_bounds__(384)
gemm_nt_few(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, int M,
            int N, int K, long long lda, long long ldw, long long ldc, int rows) {
  extern __shared__ __align__(16) float ring[];            // STAGES x (FN rows of W, `rows` rows of A)
  constexpr int FROW = FK + 4;
  const int tid = threadIdx.x, first_copy = blockDim.x - 32 * COPY_WARPS;
  const int n0 = blockIdx.x * FN;
  const int lane = tid & 31, f = lane % FN, r0 = ((tid >> 5) * (32 / FN) + lane / FN) * FR;
  const int per = (FN + rows) * FROW;
  const int slices = (K + FK - 1) / FK;
  auto copy = [&](int s) {
    if (s < slices && tid >= first_copy) {
      float* dst = ring + (s % STAGES) * per;
      for (int e = tid - first_copy; e < (FN + rows) * (FK / 4); e += 32 * COPY_WARPS) {
        const int r = e / (FK / 4), k = s * FK + e % (FK / 4) * 4;
        const bool w = r < FN;
        const int row = w ? n0 + r : r - FN;
        const bool there = k < K && row < (w ? N : M);
        const float* src = w ? W + (long long)(there ? row : 0) * ldw : A + (long long)(there ? row : 0) * lda;
        copy16(dst + r * FROW + e % (FK / 4) * 4, src + (there ? k : 0), there);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  float acc[FR];
#pragma unroll
  for (int i = 0; i < FR; ++i) acc[i] = 0.f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) copy(s);
  for (int s = 0; s < slices; ++s) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
    __syncthreads();                                       // stage s has landed; stage s - 1 is read and may be written
    copy(s + STAGES - 1);
    if (tid < first_copy) {
      const float* w = ring + (s % STAGES) * per + f * FROW;
      const float* a = ring + (s % STAGES) * per + (FN + r0) * FROW;
#pragma unroll 4
      for (int k = 0; k < FK; k += 4) {
        const float4 wv = *reinterpret_cast<const float4*>(w + k);
        float4 av[FR];
#pragma unroll
        for (int i = 0; i < FR; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * FROW + k);
#pragma unroll
        for (int i = 0; i < FR; ++i) acc[i] = fmaf(av[i].x, wv.x, acc[i]);
#pragma unroll
        for (int i = 0; i < FR; ++i) acc[i] = fmaf(av[i].y, wv.y, acc[i]);
#pragma unroll
        for (int i = 0; i < FR; ++i) acc[i] = fmaf(av[i].z, wv.z, acc[i]);
#pragma unroll
        for (int i = 0; i < FR; ++i) acc[i] = fmaf(av[i].w, wv.w, acc[i]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  const int n = n0 + f;
  if (n >= N || tid >= first_copy) return;
#pragma unroll
  for (int i = 0; i < FR; ++i)
    if (r0 + i < M) C[(long long)(r0 + i) * ldc + n] = bias ? acc[i] + bias[n] : acc[i];
}

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(THREADS)
gemm_nt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const float* __restrict__ bias, TC* __restrict__ C,
               int M, int N, int K, long long lda, long long ldw, long long ldc) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int ty = tid / 16, tx = tid % 16;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < (BM * BK) / THREADS; ++i) {
      const int idx = tid + i * THREADS;
      const int r = idx / BK, c = idx % BK;
      const int m = m0 + r, k = k0 + c;
      As[c][r] = (m < M && k < K) ? to_f(A[(long long)m * lda + k]) : 0.f;
      const int n = n0 + r;
      Ws[c][r] = (n < N && k < K) ? to_f(W[(long long)n * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      C[(long long)m * ldc + n] = from_f<TC>(v);
    }
  }
}

template <typename TA, typename TW, typename TC>
int launch(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, long long lda,
           long long ldw, long long ldc, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  gemm_nt_kernel<TA, TW, TC><<<grid, THREADS, 0, stream>>>((const TA*)A, (const TW*)W, bias, (TC*)C, M, N, K, lda,
                                                          ldw, ldc);
  return 0;
}

template <int FN, int FR, int STAGES, int FK>
int launch_few(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldw,
               long long ldc, cudaStream_t stream) {
  const int per_warp = FR * (32 / FN);                     // rows of A that a warp sums
  const int warps = (M + per_warp - 1) / per_warp;
  const int rows = warps * per_warp;
  const size_t smem = (size_t)STAGES * (FN + rows) * (FK + 4) * sizeof(float);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(gemm_nt_few<FN, FR, STAGES, FK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  gemm_nt_few<FN, FR, STAGES, FK><<<(N + FN - 1) / FN, 32 * (warps + COPY_WARPS), smem, stream>>>(A, W, bias, C, M, N, K, lda, ldw, ldc, rows);
  return 0;
}

template <int TBM, int TBN, int TM, int TN, int KS>
int launch_tile(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldw,
                long long ldc, cudaStream_t stream) {
  const dim3 grid((N + TBN - 1) / TBN, (M + TBM - 1) / TBM);
  gemm_nt_tile<TBM, TBN, TM, TN, KS><<<grid, (TBM / TM) * (TBN / TN), 0, stream>>>(A, W, bias, C, M, N, K, lda, ldw, ldc);
  return 0;
}

// 32-bit operands whose rows start on 16 bytes.
int launch_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldw,
               long long ldc, cudaStream_t stream) {
  const int sms = fmx_num_sms();
#define FMX_F32_ARGS A, W, bias, C, M, N, K, lda, ldw, ldc, stream
  if (N < 32 * sms && M <= 32) {
    // 2,048 x 8,192: M = 4 58 us (<16, 2, 5, 128> 62), M = 20 76 us (<16, 4, 4, 128> 88), M = 32 93 us (93; at 3,072 x 2,048 52 and 37)
    if (M <= 4) return launch_few<16, 1, 8, 64>(FMX_F32_ARGS);
    if (M <= 20) return launch_few<16, 2, 5, 128>(FMX_F32_ARGS);
    return launch_few<16, 4, 4, 128>(FMX_F32_ARGS);
  }
  // 16,384 x 2,048: M = 4 36 us (four rows a lane 37), M = 8 45 us (two 49), M = 20 85 us (tiles of 32 x 64 95), M = 32 125 us (95)
  if (M <= 4) return launch_few<32, 2, 4, 64>(FMX_F32_ARGS);
  if (M <= 20) return launch_few<32, 4, 4, 64>(FMX_F32_ARGS);
  if (M <= 32) return launch_tile<32, 64, 4, 4, 32>(FMX_F32_ARGS);
  // The tile that takes the shortest per k, by what an SM takes for b tiles (ns, fitted to 1 to 28 tiles an SM at M = 64 to
  // 2,048 over 16,384 x 2,048, 2,048 x 8,192 and 3,072 x 2,048): a tile alone waits for its own loads, many hide each other's.
  // Against all three tiles at M = 64 to 1,024, there and over 28,672 x 4,096, 4,096 x 14,336 and 6,144 x 4,096: the best or within 1 % of it in 24
  // of 30, at worst 15 % off (64 rows of 6,144 x 4,096: 207 us, tiles of 64 x 32 180).
  auto per_sm = [&](int bm, int bn) {
    const long long tiles = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    return (float)((tiles + sms - 1) / sms);
  };
  const float large = 46.f * per_sm(128, 64) + 16.f, middle = 25.f * per_sm(64, 64) + 10.f, small = 20.f * per_sm(64, 32) + 3.f;
  if (large < middle && large < small) return launch_tile<128, 64, 8, 8, 16>(FMX_F32_ARGS);
  if (middle <= small) return launch_tile<64, 64, 8, 4, 16>(FMX_F32_ARGS);
  return launch_tile<64, 32, 4, 4, 32>(FMX_F32_ARGS);
#undef FMX_F32_ARGS
}
}  // namespace

FMX_EXPORT int fmx_gemm_simple(const void* A, const void* W, const float* bias, void* C, int M, int N, int K,
                               long long lda, long long ldw, long long ldc, int dtype_a, int dtype_w, int dtype_c,
                               cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  if (M < 0 || N < 0 || K <= 0) return fmx_fail("fmx_gemm_simple: bad sizes M=%d N=%d K=%d", M, N, K);
  if ((long long)((M + BM - 1) / BM) > 65535) return fmx_fail("fmx_gemm_simple: M=%d is too large", M);
  const int key = dtype_a * 4 + dtype_w * 2 + dtype_c;
  if (key == 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0) {
    launch_f32((const float*)A, (const float*)W, bias, (float*)C, M, N, K, lda, ldw, ldc, stream);
    FMX_LAUNCH_CHECK();
    return 0;
  }
  switch (key) {
    case 0: launch<float, float, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream); break;
    case 4: launch<bf16, float, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream); break;
    case 5: launch<bf16, float, bf16>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream); break;
    case 6: launch<bf16, bf16, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream); break;
    case 7: launch<bf16, bf16, bf16>(A, W, bias, C, M, N, K, lda, ldw, ldc, stream); break;
    default:
      return fmx_fail("fmx_gemm_simple: no kernel for element types a=%d w=%d c=%d", dtype_a, dtype_w, dtype_c);
  }
  FMX_LAUNCH_CHECK();
  return 0;
}
