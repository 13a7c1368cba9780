// The short causal convolution in front of a recurrence, with SiLU and unit vectors per head, for bfloat16 projections: a thread
// takes four neighbouring channels and walks a strip of tokens with the last inputs in registers.
//
// Bound by memory (bfloat16 in, 32-bit out).  A block per token that reads every input once per tap, a channel at a time, stood
// at 0.6 to 0.9 TB/s; here an input is read once, 8 bytes a thread, and a channel's taps once a strip.
// 2,048 tokens, 3,072 channels 54 -> 18 us (2.2 TB/s); 1,777 tokens, 6,144 channels 78 -> 29 us (2.3 TB/s); 2,048 tokens, 6,144
// channels and 4,096 decays 113 -> 47 us; 64 single tokens, 3,072 channels 24 us in two kernels -> 3.4 us in one.
// The kernels token by token (delta_prepare, ssm_prepare, channel_delta_prepare) stay for the 32-bit path, other numbers of taps
// and channels that do not come in fours.
#pragma once
#include "conv_state.cuh"
#include "packed.cuh"

namespace {
constexpr int STRIP_TAPS = 4, STRIP_CHANNELS = 512;          // channels of a block

struct ConvStrip {
  const bf16* in;                 // [T, stride]: the convolution's channels
  long long stride;
  const float *w, *bias;          // [C, 4]; [C] or null
  const int *token_row, *row_start, *row_slot;
  float* state;                   // a slot's last inputs at conv_off, [3, C]
  long long slot_stride, conv_off;
  float* out;                     // [T, C]
  int T, C, R, max_slots, strip;
  int unit, scaled;               // channels < unit form heads made unit vectors, those < scaled times `scale`
  float scale;
  int single;                     // rows of one token each: the state moves on here
  int* status;
};

__device__ __forceinline__ void strip_bad_row(const ConvStrip& a, int r, int t) {
  if (r < 0 || r >= a.R) fmx_set_status(a.status, FMX_BAD_ROW, r, t);
  else if (a.row_slot[r] >= a.max_slots) fmx_set_status(a.status, FMX_BAD_SLOT, a.row_slot[r], t);
}

// Channels [512 block, ...) of the tokens [strip * index, ...).  LG: lanes that hold a unit head (four values each); a head's
// lanes are neighbours in one warp.
template <int LG> __device__ __forceinline__ void conv_strip(const ConvStrip& a, int index, int block) {
  const int c = block * STRIP_CHANNELS + threadIdx.x * 4;
  const bool on = c < a.C, any_unit = block * STRIP_CHANNELS < a.unit;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 w[4], bias = zero, h0 = zero, h1 = zero, h2 = zero;          // taps of four channels; the three inputs before
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = on ? load4(a.w + (long long)(c + i) * STRIP_TAPS) : zero;
  if (on && a.bias != nullptr) bias = load4(a.bias + c);
  const int t0 = index * a.strip, t1 = min(a.T, t0 + a.strip);
  int cur = -2;
  bool good = false;
  float* cs = nullptr;
  for (int t = t0; t < t1; ++t) {
    const int r = a.token_row[t];
    const float4 x = on ? load4(a.in + (long long)t * a.stride + c) : zero;
    if (r != cur) {                                   // the strip's first token, or a row's
      cur = r;
      const int slot = r >= 0 && r < a.R ? a.row_slot[r] : -1;
      good = slot >= 0 && slot < a.max_slots;
      if (!good && block == 0 && threadIdx.x == 0) strip_bad_row(a, r, t);
      if (good && on) {
        cs = a.state + (long long)slot * a.slot_stride + a.conv_off + c;
        const int first = a.row_start[r], place = t - first;
        auto before = [&](int back) {                 // the input `back` tokens before t: of this portion, or out of the slot
          return place >= back ? load4(a.in + (long long)(t - back) * a.stride + c) : load4(cs + (long long)(STRIP_TAPS - 1 + place - back) * a.C);
        };
        h0 = before(3);
        h1 = before(2);
        h2 = before(1);
      }
    }
    float4 y = bias;
    auto tap = [&](float4 v, int j) {
      auto pick = [&](const float4& q) { return j == 0 ? q.x : j == 1 ? q.y : j == 2 ? q.z : q.w; };
      y.x = fmaf(pick(w[0]), v.x, y.x); y.y = fmaf(pick(w[1]), v.y, y.y);
      y.z = fmaf(pick(w[2]), v.z, y.z); y.w = fmaf(pick(w[3]), v.w, y.w);
    };
    tap(h0, 0);
    tap(h1, 1);
    tap(h2, 2);
    tap(x, 3);
    y = make_float4(silu_f(y.x), silu_f(y.y), silu_f(y.z), silu_f(y.w));
    if (any_unit) {
      float ss = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, y.w * y.w)));
#pragma unroll
      for (int d = LG / 2; d >= 1; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
      if (c < a.unit) {
        float mul = 1.0f / sqrtf(ss + 1e-6f);
        if (c < a.scaled) mul *= a.scale;
        y = make_float4(y.x * mul, y.y * mul, y.z * mul, y.w * mul);
      }
    }
    if (on) {
      store4(a.out + (long long)t * a.C + c, good ? y : zero);
      if (a.single && good) {
        store4(cs, h1);
        store4(cs + a.C, h2);
        store4(cs + 2LL * a.C, x);
      }
    }
    h0 = h1;
    h1 = h2;
    h2 = x;
  }
}

// Does the strip kernel take these sizes?  (D: a unit head's channels, or 0 where there are none.)
inline bool strip_takes(const ConvStrip& a, int taps, int D) {
  auto on16 = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  return taps == STRIP_TAPS && a.C % 4 == 0 && a.stride % 4 == 0 && a.slot_stride % 4 == 0 && a.conv_off % 4 == 0 && ((uintptr_t)a.in & 7) == 0 &&
         on16(a.w) && (a.bias == nullptr || on16(a.bias)) && on16(a.state) && on16(a.out) && (D == 0 || D == 32 || D == 64 || D == 128);
}
// Tokens of a strip: as many as leave about eight blocks to an SM (a strip reads its channels' taps and the inputs before it once),
// at most 16; single tokens of a few rows take a block each.
inline int strip_length(int T, int blocks) {
  const int n = (int)((long long)T * blocks / (8LL * fmx_num_sms()));
  return n < 1 ? 1 : n > 16 ? 16 : n;
}
}  // namespace
