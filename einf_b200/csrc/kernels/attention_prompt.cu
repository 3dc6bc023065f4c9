// Causal attention of prompts that start in this step over keys and values of their own per head, as a latent cache's rows
// give them when its up-projections are applied to the rows (bfloat16, mma.sync, 32-bit sums and softmax).
//
// A latent cache holds one row [c | r] for all heads, and attention can run on the rows as they are, with the key
// up-projection absorbed into the queries (attention_latent.cu): 2 kv_rank + rot_dim multiply-adds a (head, query, key).
// Head by head, with keys [W_uk c | r] and values W_uv c, it is dim + rot_dim + value_size, a third of that at rows of
// 512 + 64 and heads of 128, for one more product over the rows.  That pays for a prompt that is all there: every row is
// projected once and met by all later queries.  (A portion with cached tokens before it would project those anew in
// every step, a single token would project all it sees: both stay on the rows.  Which portions of a step are which is told
// here, by q_start, tile by tile: what a prompt gets does not depend on what stands beside it.)
//
// Portions of more than 64 tokens of heads in whole 128-byte lines have the kernel on tcgen05 further down; this is the one of the
// others.  A CTA has 64 queries of one head, a warp 16 of them with its queries in registers; 64 keys a tile; the next tile's keys
// are brought while this one's values are used and the other way round.  Keys come from two places (the head's plain part
// and the rotated part that all heads share), queries too.  Three CTAs an SM hide one another's waits (two warps of 32
// rows, which read half as much shared memory, have no registers left to load ahead of their products).
//
// Measured (B200): 12 heads, keys of 128 + 64, values of 128, 2,048 tokens (16 GFLOP): 116 us, against 336 us of
// attention_latent.cu on the rows of 512 + 64 (55 GFLOP); two warps of 32 rows 184 us.
// What bounds it: the chain of a tile (products, softmax, products) in the CTAs with the most keys, three of which share
// an SM, and the reads of shared memory (92 a tile and warp, 512 bytes each, against 160 products).
#include <type_traits>

#include "mma_sync.cuh"
#include "tcgen05.cuh"

namespace einf {

constexpr int kPromptRows = 64, kPromptKeys = 64, kPromptThreads = 128;

struct HeadPromptArgs {
  const __nv_bfloat16* q_plain; long long q_plain_token, q_plain_head;     // strides in elements
  const __nv_bfloat16* q_rot; long long q_rot_token, q_rot_head;
  const __nv_bfloat16* k_plain; long long k_token, k_head;
  const __nv_bfloat16* k_rot;                                              // [tokens, rot_dim]
  const __nv_bfloat16* v; long long v_token, v_head;
  const int4* tiles;                 // request, first token, tokens (up to 128), first position
  const int* q_start;                // where given, tiles of portions that do not start at position 0 are another kernel's
  __nv_bfloat16* out;                // [tokens, heads, value_size]
  const float* sink; const float* gate;
  int heads, dim, rot_dim, value_size, window, wave;
  float scale_log2;
  int* status;                       // may be null
  int short_rows;                    // portions of up to this many tokens (0: none) are the other kernel's
};

// KEY: dim + rot_dim filled up to 128 or 192; VALUE: value_size filled up to 64 or 128.
template <int KEY, int VALUE>
__global__ void __launch_bounds__(kPromptThreads, 3)
head_prompt_attention_kernel(const __grid_constant__ HeadPromptArgs a) {
  extern __shared__ __align__(128) unsigned char prompt_smem[];
  constexpr int kKeyPitch = KEY * 2, kValuePitch = VALUE * 2;
  constexpr int kK = 0, kV = kPromptKeys * kKeyPitch;
  pdl_launch_dependents();
  int row_tile, h;
  rows_of_cta(a.wave, a.heads, &row_tile, &h);
  const int4 tile = a.tiles[row_tile >> 1];
  const int sub = (row_tile & 1) * kPromptRows;
  const int rows = min(kPromptRows, tile.z - sub);
  const int key_token = tile.y - tile.w;                  // packed index of the request's position 0
  if (rows <= 0 || (a.q_start && a.q_start[tile.x] != key_token) || (a.short_rows && (tile.w > 0 || tile.z > a.short_rows))) {
    pdl_wait();
    return;
  }
  const int t0 = tile.y + sub, pos0 = tile.w + sub;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q2 = (lane & 3) * 2;
  const uint32_t base = smem_address(prompt_smem);
  const int last_pos = pos0 + rows - 1;
  const int first_tile = a.window > 0 ? max(0, pos0 - a.window + 1) / kPromptKeys : 0, end_tile = last_pos / kPromptKeys + 1;
  pdl_wait();

  // 64 rows of a plain and a rotated part, zeros from row `count` on: a thread has one 16-byte piece of every 128-byte
  // line of four rows
  auto bring = [&](uint32_t at, auto lines_tag, const __nv_bfloat16* plain, long long plain_stride, int plain_size,
                   const __nv_bfloat16* rot, long long rot_stride, int rot_size, int count) {
    constexpr int kLines = decltype(lines_tag)::value, kPitch = 128 * kLines;
    const int r0 = threadIdx.x >> 3, piece = threadIdx.x & 7;
#pragma unroll
    for (int line = 0; line < kLines; ++line) {
      const int e = 64 * line + 8 * piece;
      const bool in_plain = e < plain_size, in_rot = !in_plain && e - plain_size < rot_size;
      const __nv_bfloat16* from = plain;
      if (in_plain) from = plain + r0 * plain_stride + e;
      else if (in_rot) from = rot + r0 * rot_stride + (e - plain_size);
      const long long step = in_plain ? 16 * plain_stride : in_rot ? 16 * rot_stride : 0;
      const uint32_t to = at + r0 * kPitch + 128 * line + ((piece ^ r0) & 7) * 16;       // rows 16 apart exchange alike
      const bool any = in_plain || in_rot;
#pragma unroll
      for (int u = 0; u < 4; ++u, from += step) {
        const bool there = any && r0 + 16 * u < count;
        cp_async16(to + u * 16 * kPitch, there ? from : plain, there ? 16 : 0);
      }
    }
  };
  using KeyLines = std::integral_constant<int, KEY / 64>;
  using ValueLines = std::integral_constant<int, VALUE / 64>;
  auto bring_keys = [&](int t) {
    const int j0 = t * kPromptKeys;
    bring(base + kK, KeyLines{}, a.k_plain + (key_token + j0) * a.k_token + h * a.k_head, a.k_token, a.dim,
          a.k_rot + (long long)(key_token + j0) * a.rot_dim, a.rot_dim, a.rot_dim, last_pos + 1 - j0);
    cp_async_commit_group();
  };
  auto bring_values = [&](int t) {
    const int j0 = t * kPromptKeys;
    bring(base + kV, ValueLines{}, a.v + (key_token + j0) * a.v_token + h * a.v_head, a.v_token, a.value_size, nullptr, 0, 0,
          last_pos + 1 - j0);
    cp_async_commit_group();
  };
  const int in8 = lane & 7, second = (lane >> 3) & 1, third = lane >> 4;
  // the queries come through the keys' place
  bring(base + kK, KeyLines{}, a.q_plain + t0 * a.q_plain_token + h * a.q_plain_head, a.q_plain_token, a.dim,
        a.q_rot + t0 * a.q_rot_token + h * a.q_rot_head, a.q_rot_token, a.rot_dim, rows);
  cp_async_commit_group();
  cp_async_wait_groups<0>();
  __syncthreads();
  uint32_t Q[KEY / 16][4];
#pragma unroll
  for (int kk = 0; kk < KEY / 16; ++kk)
    ldsm_x4(Q[kk], base + kK + swizzled(16 * warp + in8 + 8 * second, 2 * kk + third, kKeyPitch));
  __syncthreads();
  bring_keys(first_tile);
  bring_values(first_tile);

  float O[VALUE / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < VALUE / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) O[j][e] = 0.f;
  const int warp_first = pos0 + 16 * warp, warp_last = warp_first + 15;

  for (int t = first_tile; t < end_tile; ++t) {
    const int j0 = t * kPromptKeys;
    // a warp none of whose rows sees a key of the tile sits the products out
    const bool seen = j0 <= warp_last && (a.window <= 0 || j0 + kPromptKeys - 1 > warp_first - a.window);
    cp_async_wait_groups<1>();                             // the keys are there
    __syncthreads();
    float S[8][4];
    if (seen) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j][e] = 0.f;
#pragma unroll
      for (int kk = 0; kk < KEY / 16; ++kk) {
        uint32_t kf[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          ldsm_x4(kf[j], base + kK + swizzled(16 * j + in8 + 8 * third, 2 * kk + second, kKeyPitch));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          mma_bf16_16816(S[2 * j], Q[kk], kf[j][0], kf[j][1]);
          mma_bf16_16816(S[2 * j + 1], Q[kk], kf[j][2], kf[j][3]);
        }
      }
    }
    __syncthreads();                                       // the keys are used up
    if (t + 1 < end_tile) bring_keys(t + 1);
    else cp_async_commit_group();                          // an empty group: the values are always the second youngest
    if (seen) {
      const bool masks = j0 + kPromptKeys - 1 > warp_first || (a.window > 0 && j0 <= warp_last - a.window);
#pragma unroll
      for (int half = 0; half < 2; ++half) {               // rows g and g + 8 of the 16
        const int pos = warp_first + g + 8 * half;
        float top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float z = S[j][2 * half + e] * a.scale_log2;
            if (masks) {
              const int key = j0 + 8 * j + q2 + e;
              z = (key <= pos && (a.window <= 0 || key > pos - a.window)) ? z : -INFINITY;
            }
            S[j][2 * half + e] = z;
            top = fmaxf(top, z);
          }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float to = fmaxf(m[half], top);
        const float shift = to == -INFINITY ? 0.f : to;
        const float factor = exp2f(m[half] - shift);       // nothing seen so far: zero
        m[half] = to;
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float w;
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(S[j][2 * half + e] - shift));
            S[j][2 * half + e] = w;
            sum += w;
          }
        l[half] = l[half] * factor + sum;                  // this lane's share; the row's lanes are added at the end
        if (__any_sync(0xffffffffu, factor != 1.f)) {
#pragma unroll
          for (int j = 0; j < VALUE / 8; ++j) {
            O[j][2 * half] *= factor;
            O[j][2 * half + 1] *= factor;
          }
        }
      }
    }
    cp_async_wait_groups<1>();                             // the values are there
    __syncthreads();
    if (seen) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {                     // the weights are the first operand as they lie in registers
        const uint32_t P[4] = {pack_pair(S[2 * kk][0], S[2 * kk][1]), pack_pair(S[2 * kk][2], S[2 * kk][3]),
                               pack_pair(S[2 * kk + 1][0], S[2 * kk + 1][1]), pack_pair(S[2 * kk + 1][2], S[2 * kk + 1][3])};
#pragma unroll
        for (int j0v = 0; j0v < VALUE / 16; j0v += 4) {
          uint32_t vf[4][4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            ldsm_x4_trans(vf[j], base + kV + swizzled(16 * kk + in8 + 8 * second, 2 * (j0v + j) + third, kValuePitch));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            mma_bf16_16816(O[2 * (j0v + j)], P, vf[j][0], vf[j][1]);
            mma_bf16_16816(O[2 * (j0v + j) + 1], P, vf[j][2], vf[j][3]);
          }
        }
      }
    }
    __syncthreads();                                       // the values are used up
    if (t + 1 < end_tile) bring_values(t + 1);
    else cp_async_commit_group();
  }
  cp_async_wait_groups<0>();

#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int r = 16 * warp + g + 8 * half;
    float sum = l[half];
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (r >= rows) continue;
    if (a.sink) sum += exp2f(a.sink[h] * 1.4426950408889634f - m[half]);
    const long long row = (long long)(t0 + r) * a.heads + h;
    float factor = sum > 0.f ? 1.f / sum : 0.f;
    if (a.gate) factor *= a.gate[row];
    __nv_bfloat16* out = a.out + row * a.value_size;
#pragma unroll
    for (int j = 0; j < VALUE / 8; ++j) {
      const int column = 8 * j + q2;
      if (column < a.value_size)
        *reinterpret_cast<uint32_t*>(out + column) = pack_pair(O[j][2 * half] * factor, O[j][2 * half + 1] * factor);
    }
  }
}

// The same on the fifth-generation tensor cores, for heads in whole 128-byte lines (dim, rot_dim and value_size multiples of
// 64): a CTA has 128 queries of one head and takes its keys 128 at a time, in turn by two warpgroups, each with scores, sums
// and an accumulator of its own, which meet at the end.  One warp brings keys and values (TMA, two stages each), one lane of
// another issues the products: scores into the group's 128 columns of tensor memory; the group's threads (a row each)
// take them out, and put the weights, as bfloat16 pairs, into the same columns, where the second product reads them as its
// first operand.  While one group is at its softmax the other's products run.  A row's reference moves only when a tile's
// maximum is more than 2^8 above it, so that the accumulator is rarely taken out and multiplied.  In a tile of which some row
// does not see every key the warp that brings the tiles clears the values behind the request's last key (another request's) and
// those that are not finite, since zero times infinity is not zero; the rows that see the latter get them added at the end.
// Measured (B200, us, the kernel above / this one): 12 heads, keys of 128 + 64, values of 128: 2,048 tokens 124 / 32 (500
// TFLOP/s), 4,096 283 / 91, 300 18.4 / 9.9, 128 10.1 / 7.8; 14 heads of 64 + 64, values of 64, 2,048 tokens 80 / 33.  Portions of up to
// 64 tokens fill half a tile of this one at most and stay above: 40 of 30 tokens 14.8 / 31.7, one of 20 6.4 / 8.2.  What bounds it
// now: a tile's softmax, 128 exponentials a thread between two passes through tensor memory.
constexpr int kHeadThreads = 320, kHeadSlice = 128 * 64 * 2;

template <int KS, int VS>
struct HeadLayout {
  static constexpr int kQ = 0, kK = KS * kHeadSlice, kV = kK + 2 * KS * kHeadSlice, kBars = kV + 2 * VS * kHeadSlice;
  static constexpr int kShared = kBars + 8 * 17 + 24, kSums = kShared, kBytes = kSums + 4 * 128 * 4 + 1024;
};

__device__ __forceinline__ bool head_wait(uint32_t bar, uint32_t parity, int* status) {
  if (bar_test(bar, parity) || bar_poll(bar, parity)) return true;
  if (status) atomicOr(status, kStatusWaitExpired);
  return false;
}

// By a warp: takes what is not finite out of the first `real` rows of a tile of values, and everything out of the rows behind
// them; true if there was something in the former.  Looked at first, eight loads under way (a store behind each: 3.4 us).
template <int VS>
__device__ __forceinline__ bool clear_tile(unsigned char* tile, int real, int lane) {
  uint4* pieces = reinterpret_cast<uint4*>(tile) + lane;
  uint32_t any = 0;
#pragma unroll 8
  for (int e = 0; e < 32 * VS; ++e) {
    const uint4 v = pieces[32 * e];
    any |= not_finite(v.x) | not_finite(v.y) | not_finite(v.z) | not_finite(v.w);
  }
  bool found = false;
  if (__any_sync(0xffffffffu, any != 0u)) {
#pragma unroll 1
    for (int e = 0; e < 32 * VS; ++e) {
      const int row = 4 * (e & 31) + (lane >> 3);
      uint4 v = pieces[32 * e];
      const uint4 out = make_uint4(not_finite(v.x), not_finite(v.y), not_finite(v.z), not_finite(v.w));
      if (row >= real || !(out.x | out.y | out.z | out.w)) continue;
      v = make_uint4(v.x & ~((out.x >> 15) * 0xffffu), v.y & ~((out.y >> 15) * 0xffffu), v.z & ~((out.z >> 15) * 0xffffu),
                     v.w & ~((out.w >> 15) * 0xffffu));
      pieces[32 * e] = v;
      found = true;
    }
  }
  for (int c = 0; c < VS; ++c)
    for (int e = real * 8 + lane; e < 128 * 8; e += 32) reinterpret_cast<uint4*>(tile + c * kHeadSlice)[e] = make_uint4(0u, 0u, 0u, 0u);
  return found;
}

// What clear_tile took out of the keys from `first` to before `last`, added to a row of the output that this thread has written
// (seldom; a call, since the loops in the kernel's own text cost the others 1.7 us a CTA).
__device__ __noinline__ void add_not_finite(const HeadPromptArgs& a, __nv_bfloat16* out, int key_token, int first, int last, int h, float weight) {
  for (int key = first; key < last; ++key) {
    const __nv_bfloat16* v = a.v + (key_token + key) * a.v_token + h * a.v_head;
    for (int e = 0; e < a.value_size; ++e) {
      const float x = __bfloat162float(v[e]);
      if (!(fabsf(x) < INFINITY)) out[e] = __float2bfloat16_rn(__bfloat162float(out[e]) + weight * x);
    }
  }
}

template <int KS, int VS>
__global__ void __launch_bounds__(kHeadThreads, 1)
head_prompt_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr,
                           const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_kr,
                           const __grid_constant__ CUtensorMap map_v, const __grid_constant__ HeadPromptArgs a) {
  using L = HeadLayout<KS, VS>;
  constexpr int kValue = VS * 64;
  extern __shared__ unsigned char head_smem[];
  int row_tile, h;
  rows_of_cta(a.wave, a.heads, &row_tile, &h);
  const int4 tile = a.tiles[row_tile];
  const int rows = tile.z, key_token = tile.y - tile.w;
  if (rows <= 0 || (a.q_start && a.q_start[tile.x] != key_token) || (tile.w == 0 && rows <= a.short_rows)) {
    pdl_launch_dependents();
    pdl_wait();
    return;
  }
  const uint32_t raw = smem_address(head_smem), base = (raw + 1023u) & ~1023u;
  unsigned char* generic = head_smem + (base - raw);
  const uint32_t bars = base + L::kBars;
  const uint32_t q_full = bars, k_full = bars + 8, k_empty = bars + 24, v_full = bars + 40, v_empty = bars + 56, s_full = bars + 72,
                 p_full = bars + 88, o_done = bars + 104, v_clear = bars + 120, holder = bars + 136;
  volatile int* taken_out = reinterpret_cast<volatile int*>(generic + L::kBars + 140);   // values that are not finite
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pos0 = tile.w, last_pos = pos0 + rows - 1;
  const int first_tile = a.window > 0 ? max(0, pos0 - a.window + 1) / 128 : 0, n = last_pos / 128 + 1 - first_tile;
  if (tid == 0) {
    *taken_out = 0;
    bar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) {
      bar_init(k_full + 8 * s, 1);
      bar_init(k_empty + 8 * s, 1);
      bar_init(v_full + 8 * s, 1);
      bar_init(v_empty + 8 * s, 1);
      bar_init(s_full + 8 * s, 1);
      bar_init(p_full + 8 * s, 128);
      bar_init(o_done + 8 * s, 1);
      bar_init(v_clear + 8 * s, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(holder) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(generic + L::kBars + 136);
  pdl_launch_dependents();
  pdl_wait();
  const int dim_lines = a.dim / 64;
  bool ok = true;
  // some row does not see some key of a tile (the last one's keys may also be another request's)
  auto hides = [&](int i) {
    const int j0 = (first_tile + i) * 128;
    return j0 + 127 > pos0 || (a.window > 0 && j0 <= last_pos - a.window);
  };
  if (warp == 8) {
    auto bring = [&](int i) {
      const int s = i & 1, token = key_token + (first_tile + i) * 128;
      const uint32_t again = ((i >> 1) & 1) ^ 1;
      if (i >= 2) ok = ok && head_wait(k_empty + 8 * s, again, a.status);
      if (!ok) return;
      bar_expect_tx(k_full + 8 * s, KS * kHeadSlice);
      for (int c = 0; c < KS; ++c) {
        const uint32_t to = base + L::kK + (s * KS + c) * kHeadSlice;
        if (c < dim_lines) tma_2d(to, &map_k, (int)(h * a.k_head) + 64 * c, token, k_full + 8 * s);
        else tma_2d(to, &map_kr, 64 * (c - dim_lines), token, k_full + 8 * s);
      }
      if (i >= 2) ok = ok && head_wait(v_empty + 8 * s, again, a.status);
      if (!ok) return;
      bar_expect_tx(v_full + 8 * s, VS * kHeadSlice);
      for (int c = 0; c < VS; ++c)
        tma_2d(base + L::kV + (s * VS + c) * kHeadSlice, &map_v, (int)(h * a.v_head) + 64 * c, token, v_full + 8 * s);
    };
    if (lane == 0) {
      bar_expect_tx(q_full, KS * kHeadSlice);
      for (int c = 0; c < KS; ++c) {
        if (c < dim_lines) tma_2d(base + L::kQ + c * kHeadSlice, &map_q, (int)(h * a.q_plain_head) + 64 * c, tile.y, q_full);
        else tma_2d(base + L::kQ + c * kHeadSlice, &map_qr, (int)(h * a.q_rot_head) + 64 * (c - dim_lines), tile.y, q_full);
      }
      bring(0);
    }
    for (int i = 0; i < n; ++i) {
      if (i + 1 < n && lane == 0) bring(i + 1);            // before the look at tile i, which its stages do not wait for
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      if (!ok) break;
      if (!hides(i)) continue;
      const int s = i & 1;
      ok = __all_sync(0xffffffffu, head_wait(v_full + 8 * s, (i >> 1) & 1, a.status)) != 0;
      if (!ok) break;
      if (clear_tile<VS>(generic + L::kV + s * VS * kHeadSlice, last_pos + 1 - (first_tile + i) * 128, lane)) *taken_out = 1;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(v_clear + 8 * s);
    }
  } else if (warp == 9) {
    constexpr uint32_t kScores = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    constexpr uint32_t kMix = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(kValue >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    ok = head_wait(q_full, 0, a.status);
    auto scores = [&](int i) {
      const int s = i & 1, turn = i >> 1;
      ok = ok && head_wait(k_full + 8 * s, turn & 1, a.status);
      if (turn > 0) ok = ok && head_wait(o_done + 8 * s, (turn - 1) & 1, a.status);   // the group's weights are used up
      if (!ok || lane != 0) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < KS; ++c) {
        const uint64_t q = desc_k_major(base + L::kQ + c * kHeadSlice), k = desc_k_major(base + L::kK + (s * KS + c) * kHeadSlice);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma_ss(tmem + 128 * s, desc_advance(q, kk * 32), desc_advance(k, kk * 32), kScores, c > 0 || kk > 0);
      }
      mma_commit(k_empty + 8 * s);
      mma_commit(s_full + 8 * s);
    };
    if (n > 0) scores(0);
    uint32_t cleared = 0;                                  // parity of either stage's tiles that hide something, so far
    for (int i = 0; i < n; ++i) {
      const int s = i & 1, turn = i >> 1;
      if (i + 1 < n) scores(i + 1);
      ok = ok && (hides(i) ? head_wait(v_clear + 8 * s, cleared >> s & 1, a.status) : head_wait(v_full + 8 * s, turn & 1, a.status));
      if (hides(i)) cleared ^= 1u << s;
      __syncwarp();
      ok = ok && head_wait(p_full + 8 * s, turn & 1, a.status);
      if (ok && lane == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t v = desc_mn_major(base + L::kV + s * VS * kHeadSlice, kHeadSlice);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) mma_ts(tmem + 256 + 128 * s, tmem + 128 * s + kk * 8, desc_advance(v, kk * 2048), kMix, turn > 0 || kk > 0);
        mma_commit(v_empty + 8 * s);
        mma_commit(o_done + 8 * s);
      }
      __syncwarp();
    }
  }
  float m = -INFINITY, l = 0.f;
  const int group = (warp >> 2) & 1, r = (warp & 3) * 32 + lane;
  const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16), mine = lanes + 128 * group, mixed = lanes + 256 + 128 * group;
  const int turns = (n - group + 1) >> 1;
  if (warp < 8) {
    const int pos = pos0 + r;
    for (int turn = 0; turn < turns && ok; ++turn) {
      ok = head_wait(s_full + 8 * group, turn & 1, a.status);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int j0 = (first_tile + 2 * turn + group) * 128;
      float z[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(mine + 32 * c, z + 32 * c);
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_wait32(z + 32 * c);
      if (j0 + 127 > pos0 || (a.window > 0 && j0 <= last_pos - a.window)) {
        const int to = pos - j0, from = a.window > 0 ? to - a.window : -1;        // visible: from < key <= to
#pragma unroll
        for (int e = 0; e < 128; ++e) z[e] = e <= to && e > from ? z[e] : -INFINITY;
      }
      float top = -INFINITY;
#pragma unroll
      for (int e = 0; e < 128; ++e) top = fmaxf(top, z[e]);
      top *= a.scale_log2;
      const bool moves = top > m + 8.f || (m == -INFINITY && top > -INFINITY);
      if (__any_sync(0xffffffffu, moves)) {
        const float factor = moves ? exp2f(m - top) : 1.f;       // nothing seen so far: zero
        if (moves) m = top;
        l *= factor;
        if (turn > 0) {                                           // the scores' arrival says that the last product is over
#pragma unroll
          for (int c = 0; c < kValue / 32; ++c) {
            float o[32];
            tmem_ld32(mixed + 32 * c, o);
            tmem_ld_wait32(o);
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] *= factor;
            tmem_st32(mixed + 32 * c, o);
          }
        }
      }
      const float shift = m == -INFINITY ? 0.f : m;
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pairs[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float x = fast_exp2(fmaf(z[32 * c + 2 * e], a.scale_log2, -shift)), y = fast_exp2(fmaf(z[32 * c + 2 * e + 1], a.scale_log2, -shift));
          sum += x + y;
          pairs[e] = pack_pair(x, y);
        }
        tmem_st16(mine + 16 * c, pairs);
      }
      l += sum;
      tmem_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      bar_arrive(p_full + 8 * group);
    }
    if (turns > 0) ok = ok && head_wait(o_done + 8 * group, (turns - 1) & 1, a.status);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    float* shared = reinterpret_cast<float*>(generic + L::kSums);
    shared[group * 128 + r] = m;
    shared[256 + group * 128 + r] = l;
  }
  __syncthreads();
  float factor = 0.f;
  bool seen = false;
  float* half = reinterpret_cast<float*>(generic + L::kK);        // the second group's share: every load and product is over
  constexpr int kPitch = kValue + 1;
  static_assert(128 * kPitch * 4 <= (2 * KS + 2 * VS) * kHeadSlice, "the share fits the keys' and values' place");
  if (warp < 8) {
    const float* shared = reinterpret_cast<const float*>(generic + L::kSums);
    const float m0 = shared[r], m1 = shared[128 + r], top = fmaxf(m0, m1), at = top == -INFINITY ? 0.f : top;
    float total = shared[256 + r] * exp2f(m0 - at) + shared[384 + r] * exp2f(m1 - at);
    if (a.sink) total += exp2f(a.sink[h] * 1.4426950408889634f - top);
    // a sum that is not a number is the row's result: only what has seen nothing, or nothing of any weight, is zero
    seen = m != -INFINITY || l != 0.f;
    factor = seen && total != 0.f ? exp2f(m - at) / total : 0.f;
    if (a.gate && r < rows) factor *= a.gate[(long long)(tile.y + r) * a.heads + h];
    if (group == 1 && turns > 0) {
#pragma unroll
      for (int c = 0; c < kValue / 32; ++c) {
        float o[32];
        tmem_ld32(mixed + 32 * c, o);
        tmem_ld_wait32(o);
#pragma unroll
        for (int e = 0; e < 32; ++e) half[r * kPitch + 32 * c + e] = seen ? o[e] * factor : 0.f;
      }
    }
  }
  __syncthreads();
  if (warp < 4) {
    __nv_bfloat16* out = a.out + ((long long)(tile.y + r) * a.heads + h) * kValue;
#pragma unroll
    for (int c = 0; c < kValue / 32; ++c) {
      float o[32];
      tmem_ld32(mixed + 32 * c, o);
      tmem_ld_wait32(o);
      uint32_t pairs[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        float x = seen ? o[2 * e] * factor : 0.f, y = seen ? o[2 * e + 1] * factor : 0.f;
        if (n > 1) {
          x += half[r * kPitch + 32 * c + 2 * e];
          y += half[r * kPitch + 32 * c + 2 * e + 1];
        }
        pairs[e] = pack_pair(x, y);
      }
      if (r < rows) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          *reinterpret_cast<uint4*>(out + 32 * c + 8 * e) = make_uint4(pairs[4 * e], pairs[4 * e + 1], pairs[4 * e + 2], pairs[4 * e + 3]);
      }
    }
    if (*taken_out && r < rows)
      for (int i = 0; i < n; ++i) {
        const int j0 = (first_tile + i) * 128;
        if (hides(i))
          add_not_finite(a, out, key_token, a.window > 0 ? max(j0, pos0 + r - a.window + 1) : j0, min(j0 + 128, pos0 + r + 1), h,
                         a.gate ? a.gate[(long long)(tile.y + r) * a.heads + h] : 1.f);
      }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 9) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// rows x cols bfloat16, unit stride along cols, rows `stride` elements apart, box of (64 cols x 128 rows), 128-byte swizzle
static int head_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long stride) {
  EncodeTiledFn encode = encode_tiled();
  if (!encode) return (int)cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)stride * 2};
  cuuint32_t box[2] = {64, 128};
  cuuint32_t element_strides[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, element_strides,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <int KS, int VS>
static int launch_head_tcgen05(const HeadPromptArgs& a, int tokens, int num_tiles, cudaStream_t stream) {
  CUtensorMap q, qr, k, kr, v;
  int e = head_map(&q, a.q_plain, tokens, (a.heads - 1) * a.q_plain_head + a.dim, a.q_plain_token);
  if (!e) e = head_map(&qr, a.q_rot, tokens, (a.heads - 1) * a.q_rot_head + a.rot_dim, a.q_rot_token);
  if (!e) e = head_map(&k, a.k_plain, tokens, (a.heads - 1) * a.k_head + a.dim, a.k_token);
  if (!e) e = head_map(&kr, a.k_rot, tokens, a.rot_dim, a.rot_dim);
  if (!e) e = head_map(&v, a.v, tokens, (a.heads - 1) * a.v_head + a.value_size, a.v_token);
  if (e) return e;
  auto kernel = head_prompt_tcgen05_kernel<KS, VS>;
  constexpr int kBytes = HeadLayout<KS, VS>::kBytes;
  const cudaError_t set = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (set != cudaSuccess) return (int)set;
  return (int)launch_pdl(kernel, dim3(num_tiles * a.heads), dim3(kHeadThreads), kBytes, stream, q, qr, k, kr, v, a);
}

// Cached rows of the step's tokens, taken apart: rows[t] = the first `first` elements of the row in slot t, rest[t] the next
// `second` (multiples of eight; a token without a slot gets zeros).
__global__ void __launch_bounds__(256)
latent_rows_kernel(const __nv_bfloat16* __restrict__ cache, const int* __restrict__ slots, long long num_rows, int row_size,
                   __nv_bfloat16* __restrict__ rows, int first, __nv_bfloat16* __restrict__ rest, int second, int tokens) {
  pdl_launch_dependents();
  pdl_wait();
  const int pieces = (first + second) / 8;
  const long long total = (long long)tokens * pieces;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / pieces), e = 8 * (int)(i - (long long)t * pieces);
    const int slot = slots[t];
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (slot >= 0 && slot < num_rows) v = *reinterpret_cast<const uint4*>(cache + (long long)slot * row_size + e);
    __nv_bfloat16* to = e < first ? rows + (long long)t * first + e : rest + (long long)t * second + (e - first);
    *reinterpret_cast<uint4*>(to) = v;
  }
}

template <int KEY, int VALUE>
static cudaError_t launch_head_prompt(const HeadPromptArgs& a, int num_tiles, cudaStream_t stream) {
  auto kernel = head_prompt_attention_kernel<KEY, VALUE>;
  constexpr int kBytes = kPromptKeys * (KEY + VALUE) * 2;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return e;
  return launch_pdl(kernel, dim3(2 * num_tiles * a.heads), dim3(kPromptThreads), kBytes, stream, a);
}

}  // namespace einf

using namespace einf;

extern "C" int einf_latent_rows(const void* cache, const int* slots, long long num_rows, int row_size, void* rows, int first,
                                void* rest, int second, int tokens, cudaStream_t stream) {
  if (tokens == 0) return 0;
  if (first % 8 || second % 8 || row_size % 8 || first <= 0 || second < 0 || first + second > row_size ||
      (((uintptr_t)cache | (uintptr_t)rows | (uintptr_t)rest) & 15))
    return (int)cudaErrorInvalidValue;
  const long long ctas = ((long long)tokens * ((first + second) / 8) + 255) / 256;
  return (int)launch_pdl(latent_rows_kernel, dim3((unsigned)(ctas < 148 * 8 ? ctas : 148 * 8)), dim3(256), 0, stream,
                         (const __nv_bfloat16*)cache, slots, num_rows, row_size, (__nv_bfloat16*)rows, first,
                         (__nv_bfloat16*)rest, second, tokens);
}

// `tensor_memory`: by the kernel on tcgen05 (sizes multiples of 64, rot_dim and scale above 0), `short_rows`: of it and the other kernel,
// the other one has the portions of up to that many tokens and this one the longer ones (0: the kernel has all).
// Portions that start at position 0 in this step, their tokens packed one after the other; with `q_start`, the requests' first
// tokens, `tiles` of other portions are left out (without it there must be none).  Sizes and
// strides in multiples of eight elements, pointers on 16-byte borders; dim + rot_dim up to 192, value_size up to 128.
// `wave`: multiprocessors of the device.
extern "C" int einf_head_prompt_attention(const void* q_plain, long long q_plain_token, long long q_plain_head,
                                          const void* q_rot, long long q_rot_token, long long q_rot_head, const void* k_plain,
                                          long long k_token, long long k_head, const void* k_rot, const void* v,
                                          long long v_token, long long v_head, const int* tiles, int num_tiles,
                                          const int* q_start, void* out,
                                          const float* sink, const float* gate, int heads, int dim, int rot_dim,
                                          int value_size, int window, float scale, int wave, int tokens, int tensor_memory, int short_rows, int* status,
                                          cudaStream_t stream) {
  if (num_tiles == 0) return 0;
  const long long strides = q_plain_token | q_plain_head | q_rot_token | q_rot_head | k_token | k_head | v_token | v_head;
  if (heads <= 0 || 2ll * num_tiles * heads > 0x7fffffff || dim <= 0 || rot_dim < 0 || dim + rot_dim > 192 ||
      value_size <= 0 || value_size > 128 || ((dim | rot_dim | value_size) & 7) || (strides & 7) || wave <= 0 ||
      (((uintptr_t)q_plain | (uintptr_t)q_rot | (uintptr_t)k_plain | (uintptr_t)k_rot | (uintptr_t)v | (uintptr_t)out |
        (uintptr_t)tiles) & 15))
    return (int)cudaErrorInvalidValue;
  HeadPromptArgs a;
  a.q_plain = (const __nv_bfloat16*)q_plain; a.q_plain_token = q_plain_token; a.q_plain_head = q_plain_head;
  a.q_rot = (const __nv_bfloat16*)q_rot; a.q_rot_token = q_rot_token; a.q_rot_head = q_rot_head;
  a.k_plain = (const __nv_bfloat16*)k_plain; a.k_token = k_token; a.k_head = k_head;
  a.k_rot = (const __nv_bfloat16*)k_rot;
  a.v = (const __nv_bfloat16*)v; a.v_token = v_token; a.v_head = v_head;
  a.tiles = (const int4*)tiles; a.q_start = q_start; a.out = (__nv_bfloat16*)out; a.sink = sink; a.gate = gate;
  a.heads = heads; a.dim = dim; a.rot_dim = rot_dim; a.value_size = value_size; a.window = window; a.wave = wave;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.status = status;
  a.short_rows = short_rows;
  if (tensor_memory) {
    if (dim % 64 || rot_dim % 64 || rot_dim == 0 || value_size % 64 || tokens <= 0 || !(scale > 0.f)) return (int)cudaErrorInvalidValue;
    if (dim + rot_dim == 128)
      return value_size == 64 ? launch_head_tcgen05<2, 1>(a, tokens, num_tiles, stream) : launch_head_tcgen05<2, 2>(a, tokens, num_tiles, stream);
    return value_size == 64 ? launch_head_tcgen05<3, 1>(a, tokens, num_tiles, stream) : launch_head_tcgen05<3, 2>(a, tokens, num_tiles, stream);
  }
  if (dim + rot_dim <= 128)
    return (int)(value_size <= 64 ? launch_head_prompt<128, 64>(a, num_tiles, stream)
                                  : launch_head_prompt<128, 128>(a, num_tiles, stream));
  return (int)(value_size <= 64 ? launch_head_prompt<192, 64>(a, num_tiles, stream)
                                : launch_head_prompt<192, 128>(a, num_tiles, stream));
}
