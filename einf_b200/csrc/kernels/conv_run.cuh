// A short causal convolution per channel over runs of tokens: a thread has four channels of eight neighbouring tokens,
// brings the eight rows and the three before them once (16-byte or 8-byte loads, all in flight together) and keeps the
// window in registers, where a thread per element reads every row `taps` times, four bytes or two at a time, behind a 64-bit
// division.  For up to four taps; the additions are those of the per-element kernels, in their order.
#pragma once

#include "common.cuh"

namespace einf {

constexpr int kRunTokens = 8, kRunTaps = 4;
constexpr long long kRunElements = 1 << 19;      // of a launch above which runs are the faster way (einf_conv_silu)

template <typename T>
__device__ __forceinline__ float4 load_quad(const T* p) {
  if constexpr (sizeof(T) == 4) {
    return *reinterpret_cast<const float4*>(p);
  } else {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                       __uint_as_float(raw.y & 0xffff0000u));
  }
}
template <typename T>
__device__ __forceinline__ void store_quad(T* p, float4 v) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
  }
}

// finish(token, input, sum): what becomes of a token's sum (`input` its own row); start(): what the sum starts from, or the
// input itself with kFromInput.  `state` rows are the taps - 1 inputs before a request's tokens, oldest first.  `updates`: the
// step has one request, whose first tokens, and with them all that reads its state row, are the first run's: its thread then
// leaves the request's last taps - 1 inputs there (rows may go on behind its end, q_start[1]; of more requests a run may begin behind another's first token: a kernel behind
// this one does it).
template <typename T, bool kFromInput, typename Finish>
__device__ __forceinline__ void conv_run(const T* __restrict__ in, long long in_stride, int c, int t0, int num_tokens, int taps,
                                         const float* __restrict__ weight, float4 bias, float4 start,
                                         float* state, long long state_stride, int channels,
                                         const int* __restrict__ seq_of_token, const int* __restrict__ q_start,
                                         const int* __restrict__ state_slots, int num_slots, bool updates,
                                         Finish finish) {
  constexpr int kRows = kRunTokens + kRunTaps - 1;
  const int n = min(kRunTokens, num_tokens - t0);
  float4 x[kRows];                                       // x[i]: the input of token t0 - 3 + i
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int t = t0 - (kRunTaps - 1) + i;
    x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t >= 0 && t < num_tokens) {
      x[i] = load_quad(in + (long long)t * in_stride + c);
      x[i].x += bias.x;
      x[i].y += bias.y;
      x[i].z += bias.z;
      x[i].w += bias.w;
    }
  }
  int request[kRunTokens], first[kRunTokens];
#pragma unroll
  for (int k = 0; k < kRunTokens; ++k) request[k] = k < n ? seq_of_token[t0 + k] : -1;
#pragma unroll
  for (int k = 0; k < kRunTokens; ++k) first[k] = k < n ? q_start[request[k]] : 0;
  float w[4][kRunTaps];                                  // the last `taps` of kRunTaps places
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int j = 0; j < kRunTaps; ++j)
      w[e][j] = j >= kRunTaps - taps ? weight[(long long)(c + e) * taps + j - (kRunTaps - taps)] : 0.f;
#pragma unroll
  for (int k = 0; k < kRunTokens; ++k) {
    if (k >= n) break;
    const int t = t0 + k;
    float4 acc = kFromInput ? x[k + kRunTaps - 1] : start;
#pragma unroll
    for (int j = 0; j < kRunTaps; ++j) {
      if (j < kRunTaps - taps) continue;
      const int u = t - (kRunTaps - 1) + j;
      float4 v = x[k + j];
      if (u < first[k]) {                                // before the request's tokens of the step
        const int slot = state_slots[request[k]];
        v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (slot >= 0 && slot < num_slots) {
          const float* row = state + (long long)slot * state_stride + (long long)(taps - 1 - (first[k] - u)) * channels + c;
          v = make_float4(row[0], row[1], row[2], row[3]);
        }
      }
      acc.x = fmaf(w[0][j], v.x, acc.x);
      acc.y = fmaf(w[1][j], v.y, acc.y);
      acc.z = fmaf(w[2][j], v.z, acc.z);
      acc.w = fmaf(w[3][j], v.w, acc.w);
    }
    finish(t, acc);
  }
  if (!updates || t0 != 0) return;
  const int slot = state_slots[0], keep = taps - 1, count = q_start[1] - q_start[0];
  if (slot < 0 || slot >= num_slots || count <= 0) return;
  float* rows = state + (long long)slot * state_stride + c;
  float4 fresh[kRunTaps - 1];
#pragma unroll
  for (int u = 0; u < kRunTaps - 1; ++u) {
    if (u >= keep) break;
    const int rel = count - keep + u;                    // below zero: of the old state, by a portion shorter than it
    if (rel >= 0) {
      const float4 v = load_quad(in + (long long)(q_start[0] + rel) * in_stride + c);
      fresh[u] = make_float4(v.x + bias.x, v.y + bias.y, v.z + bias.z, v.w + bias.w);
    } else {
      const float* row = rows + (long long)(u + count) * channels;
      fresh[u] = make_float4(row[0], row[1], row[2], row[3]);
    }
  }
#pragma unroll
  for (int u = 0; u < kRunTaps - 1; ++u) {
    if (u >= keep) break;
    float* row = rows + (long long)u * channels;
    row[0] = fresh[u].x;
    row[1] = fresh[u].y;
    row[2] = fresh[u].z;
    row[3] = fresh[u].w;
  }
}

}  // namespace einf
