// Retention: linear attention with one fixed decay per head and no softmax or denominator.
//
// Per head h, with q, k (size D) and v (size P), a token does
//     S <- decay_h S + k v^T;   o = S^T q,
// S [D, P] in 32-bit in a state slot of the request, carried from step to step.  That is the state-space
// recurrence of ssm.cu with a step size of 1, a decay that no token changes, as many groups as heads and no skip
// term, so the recurrence itself runs on ssm_scan; what is here stands in front of it and behind it.
//
//   retention_prepare    per token: q and k of every head rotated over their first `rot` dimensions (dimension i
//                        paired with i + rot/2; angle, sine and cosine in 32-bit), k multiplied by `k_scale` after
//                        the rotation; out [T, C] in 32-bit, C = H*P + 2*H*D, laid out as the scan takes its
//                        operands: v | k | q; and per head a step size of 1 and the head's decay, [T, 2H].
//   retention_gate_norm  o divided by its root mean square over the head (no weight), times silu(gate), out in the
//                        run's type: the kernels of head_norm.cu.
//
// Everything is 32-bit but the projection that comes in and the activations that go out.
#include <math.h>
#include "packed.cuh"

extern "C" int fmx_head_norm_gate(const float* o, const void* gate, long long gate_stride, int g_dtype, const float* w, void* out,
                                  long long out_stride, int dtype, int T, int H, int Dv, float eps, int silu, int w_stride, const float* nq,
                                  const float* gates, cudaStream_t stream);

namespace {
// proj [T, stride]: q (H*D) | k (H*D) | v (H*P)
template <typename T>
__global__ void __launch_bounds__(128)
retention_prepare_kernel(const T* proj, long long stride, const int* positions, const float* __restrict__ inv_freq,
                         const float* __restrict__ decay, float* out_xbc, float* out_dd, int H, int D, int P, int rot,
                         float k_scale) {
  extern __shared__ float smem[];               // [rot/2] sines, [rot/2] cosines
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x;
  const int half = rot / 2;
  float* sn = smem;
  float* cs = smem + half;
  const float pos = (float)positions[t];
  for (int j = threadIdx.x; j < half; j += blockDim.x) sincosf(pos * inv_freq[j], &sn[j], &cs[j]);
  __syncthreads();
  const T* row = proj + (long long)t * stride;
  const int inner = H * P, HD = H * D, C = inner + 2 * HD;
  float* ox = out_xbc + (long long)t * C;
  for (int e = threadIdx.x; e < inner; e += blockDim.x) ox[e] = to_f(row[2 * HD + e]);
  // one thread per (q or k, head, pair or unrotated dimension)
  const int per_head = D - half;                 // `half` pairs and D - rot dimensions that pass
  for (int it = threadIdx.x; it < 2 * H * per_head; it += blockDim.x) {
    const int which = it / (H * per_head);       // 0: q, 1: k
    const int rem = it - which * H * per_head;
    const int h = rem / per_head, j = rem - h * per_head;
    const T* src = row + (long long)which * HD + (long long)h * D;
    float* dst = ox + inner + (long long)(which == 0 ? HD : 0) + (long long)h * D;      // k first, then q
    const float mul = which == 0 ? 1.0f : k_scale;
    if (j < half) {
      float x, y;
      rope_pair(to_f(src[j]), to_f(src[j + half]), sn[j], cs[j], x, y);
      dst[j] = x * mul;
      dst[j + half] = y * mul;
    } else {
      const int e = j + half;
      dst[e] = to_f(src[e]) * mul;
    }
  }
  float* od = out_dd + (long long)t * 2 * H;
  for (int h = threadIdx.x; h < H; h += blockDim.x) {
    od[h] = 1.0f;
    od[H + h] = decay[h];
  }
}


// The same four values a thread, where heads, pairs and rows come in fours: bound by memory (1,531 tokens of 32 heads of 64 + 64
// values, 32-bit in and out: 26 -> 18 us).
template <typename T>
__global__ void __launch_bounds__(128)
retention_prepare_vec_kernel(const T* proj, long long stride, const int* positions, const float* __restrict__ inv_freq,
                             const float* __restrict__ decay, float* out_xbc, float* out_dd, int H, int D, int P, int rot,
                             float k_scale) {
  extern __shared__ __align__(16) float smem[];               // [rot/2] sines, [rot/2] cosines
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, half = rot / 2, inner = H * P, HD = H * D;
  float *sn = smem, *cs = smem + half;
  const float pos = (float)positions[t];
  for (int j = threadIdx.x; j < half; j += 128) sincosf(pos * inv_freq[j], &sn[j], &cs[j]);
  const T* row = proj + (long long)t * stride;
  float* ox = out_xbc + (long long)t * (inner + 2 * HD);
#pragma unroll 4
  for (int e = threadIdx.x * 4; e < inner; e += 512) store4(ox + e, load4(row + 2 * HD + e));
  __syncthreads();
  const int quads = (D - half) / 4;              // of a head: half / 4 of four pairs, then those of four values that pass
#pragma unroll 2
  for (int it = threadIdx.x; it < 2 * H * quads; it += 128) {
    const int h = it / quads, j = (it - h * quads) * 4;          // heads of q, then of k
    const float mul = h < H ? 1.0f : k_scale;
    const T* src = row + (long long)h * D;
    float* dst = ox + inner + (long long)(h < H ? h + H : h - H) * D;      // k first, then q
    auto put = [&](float* to, float4 v) { store4(to, make_float4(v.x * mul, v.y * mul, v.z * mul, v.w * mul)); };
    if (j < half) {
      const float4 a = load4(src + j), b = load4(src + j + half), s4 = load4(sn + j), c4 = load4(cs + j);
      float4 x, y;
      rope_pair(a.x, b.x, s4.x, c4.x, x.x, y.x);
      rope_pair(a.y, b.y, s4.y, c4.y, x.y, y.y);
      rope_pair(a.z, b.z, s4.z, c4.z, x.z, y.z);
      rope_pair(a.w, b.w, s4.w, c4.w, x.w, y.w);
      put(dst + j, x);
      put(dst + j + half, y);
    } else {
      put(dst + j + half, load4(src + j + half));
    }
  }
  float* od = out_dd + (long long)t * 2 * H;
  for (int h = threadIdx.x; h < H; h += 128) {
    od[h] = 1.0f;
    od[H + h] = decay[h];
  }
}
}  // namespace

// rot = 0: nothing is rotated (inv_freq may then be null).  dtype: the projection's type.
FMX_EXPORT int fmx_retention_prepare(const void* proj, long long stride, int dtype, const int* positions, const float* inv_freq,
                                     const float* decay, float* out_xbc, float* out_dd, int T, int H, int D, int P, int rot,
                                     float k_scale, cudaStream_t stream) {
  if (T == 0) return 0;
  if (T < 0 || H <= 0 || D <= 0 || P <= 0 || rot < 0 || rot > D || (rot & 1))
    return fmx_fail("fmx_retention_prepare: bad sizes T=%d H=%d D=%d P=%d rot=%d", T, H, D, P, rot);
  if (rot > 0 && inv_freq == nullptr) return fmx_fail("fmx_retention_prepare: rot=%d needs a frequency table", rot);
  if (stride < 2LL * H * D + (long long)H * P) return fmx_fail("fmx_retention_prepare: rows too narrow");
  const size_t smem = (size_t)rot * sizeof(float);
  if (D % 4 == 0 && P % 4 == 0 && rot % 8 == 0 && stride % 4 == 0 && ((uintptr_t)out_xbc & 15) == 0 && (dtype == FMX_F32 || dtype == FMX_BF16) &&
      ((uintptr_t)proj & (dtype == FMX_F32 ? 15 : 7)) == 0) {
    if (dtype == FMX_F32)
      fmx_launch(retention_prepare_vec_kernel<float>, dim3(T), dim3(128), smem, stream, (const float*)proj, stride, positions, inv_freq,
                 decay, out_xbc, out_dd, H, D, P, rot, k_scale);
    else
      fmx_launch(retention_prepare_vec_kernel<bf16>, dim3(T), dim3(128), smem, stream, (const bf16*)proj, stride, positions, inv_freq,
                 decay, out_xbc, out_dd, H, D, P, rot, k_scale);
    FMX_LAUNCH_CHECK();
    return 0;
  }
  if (dtype == FMX_F32)
    fmx_launch(retention_prepare_kernel<float>, dim3(T), dim3(128), smem, stream, (const float*)proj, stride, positions, inv_freq,
               decay, out_xbc, out_dd, H, D, P, rot, k_scale);
  else if (dtype == FMX_BF16)
    fmx_launch(retention_prepare_kernel<bf16>, dim3(T), dim3(128), smem, stream, (const bf16*)proj, stride, positions, inv_freq,
               decay, out_xbc, out_dd, H, D, P, rot, k_scale);
  else
    return fmx_fail("fmx_retention_prepare: unknown dtype %d", dtype);
  FMX_LAUNCH_CHECK();
  return 0;
}

// o [T, H*P] 32-bit; gate rows of g_stride elements of type g_dtype; out rows of out_stride elements of type dtype.
FMX_EXPORT int fmx_retention_gate_norm(const float* o, const void* gate, long long g_stride, int g_dtype, void* out,
                                       long long out_stride, int dtype, int T, int H, int P, float eps, cudaStream_t stream) {
  return fmx_head_norm_gate(o, gate, g_stride, g_dtype, nullptr, out, out_stride, dtype, T, H, P, eps, 1, 0, nullptr, nullptr, stream);
}
