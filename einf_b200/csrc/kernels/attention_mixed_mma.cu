// Score-mixing attention (the statement is at the top of attention_mixed.cu) of bfloat16 prompt portions with the mixing in
// the queries.  The mixed score of head h,
//   sum_g talk[h, g] (scale q_g . k_(kv of g) - slope_g distance),
// is a score of its own: with q'_(h, c) = scale sum_(g reads key head c) talk[h, g] q_g and slope'_h = sum_g talk[h, g] slope_g
// it is sum_c q'_(h, c) . k_c - slope'_h distance, one query [q'_(h, 0) | q'_(h, 1) ..] against the key heads' rows end to end.
// So the heads meet in the queries, once a query, and not in every score (heads^2 FMAs a key, which with the exchange of all
// heads' scores through shared memory bounded the kernel of attention_mixed_tiled.cu), and a head's softmax and values
// are those of plain attention.  q' is 32-bit and enters the products as three bfloat16 parts (mma_sync.cuh).  The weights
// of up to 16 heads' prompts enter the second product as two, as in the tensor-core kernel of attention_mixed_tiled.cu;
// those of more heads and of single tokens, whose kernels there hold them in 32 bits, as three, whose sums are added to
// the output by rounded additions.  Scores, sums and the output are 32-bit.
//
// A CTA has 64 queries of one head, a warp 16 of them; 64 keys a tile; the next tile's keys are brought while this one's
// values are used and the other way round.  The parts of q' stay in shared memory: in registers (96 of them) they leave two
// CTAs an SM and no room for sums that do not wait for one another.  Takes key heads of together up to 128 elements (a
// multiple of 16 each) and value heads up to 64 or 128 (a multiple of 8).
//
// Measured (B200): 14 heads of 64 on 2 key heads, window 1,024, 2,048 tokens: 283 -> 117 us (with q' in registers 163); 32
// heads of 32 on 4, 1,024 tokens: 685 -> 136 us (119 with weights of two parts).  The tensor pipe is active 40 and 31 % of the
// time, a scheduler issues in 46 % of its cycles: the rest is the softmax between the products and what a tile's four
// barriers cost three CTAs an SM.
#include <type_traits>

#include "mma_sync.cuh"

namespace einf {

constexpr int kMixRows = 64, kMixKeys = 64, kMixThreads = 128;
constexpr int kMixKeySize = 128;                       // key heads end to end, filled up

struct MixArgs {
  const __nv_bfloat16* q;            // [tokens, heads, dim]
  const __nv_bfloat16* k_cache; const __nv_bfloat16* v_cache;
  const int* block_table; int table_width;
  const int4* tiles;                 // request, first token, tokens (up to 128), first position
  __nv_bfloat16* out;                // [tokens, heads, vdim]
  const float* slopes; const float* talk; const float* sink;
  int* status;
  int heads, kv_heads, dim, vdim, page_size, num_pages, window, wave;
  float scale_log2, out_scale;
};

// Three parts of q', a tile's keys, its values.
template <int VALUE>
constexpr int kMixSmem = 3 * kMixRows * kMixKeySize * 2 + kMixKeys * (kMixKeySize + VALUE) * 2;

// Weights x and y as PARTS pairs of bfloat16, largest first: two are 16 bits of each, three all 24.
template <int PARTS>
__device__ __forceinline__ void split_weights(float x, float y, uint32_t (&part)[PARTS][4], int e) {
#pragma unroll
  for (int p = 0; p < PARTS; ++p) {
    part[p][e] = pack_pair(x, y);
    x -= low_bf16(part[p][e]);
    y -= high_bf16(part[p][e]);
  }
}

// O += P V of 16 keys for four column tiles, P in three parts: as mma_parts does it, the tiles side by side.
__device__ __forceinline__ void add_weighted(float (*O)[4], const uint32_t (&P)[3][4], const uint32_t (&vf)[2][4]) {
  float sum[4][4];
#pragma unroll
  for (int p = 2; p >= 0; --p)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (p == 2) mma_bf16_16816_zero(sum[j], P[p], vf[j >> 1][2 * (j & 1)], vf[j >> 1][2 * (j & 1) + 1]);
      else mma_bf16_16816(sum[j], P[p], vf[j >> 1][2 * (j & 1)], vf[j >> 1][2 * (j & 1) + 1]);
    }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) O[j][e] += sum[j][e];
}

// VALUE: vdim filled up to 64 or 128; PARTS: of the weights.
template <int VALUE, int PARTS>
__global__ void __launch_bounds__(kMixThreads, VALUE <= 64 ? 3 : 2)
mixed_prompt_attention_kernel(const __grid_constant__ MixArgs a) {
  extern __shared__ __align__(128) unsigned char mix_smem[];
  __shared__ int places[2][kMixKeys];                  // of a tile's keys: the page's first row of head 0 + slot in it, -1: none
  constexpr int kKeyPitch = kMixKeySize * 2, kValuePitch = VALUE * 2;
  constexpr int kQPart = kMixRows * kKeyPitch, kK = 3 * kQPart, kV = kK + kMixKeys * kKeyPitch, kSteps = kMixKeySize / 16;
  pdl_launch_dependents();
  int row_tile, h;
  rows_of_cta(a.wave, a.heads, &row_tile, &h);
  const int4 tile = a.tiles[row_tile >> 1];
  const int sub = (row_tile & 1) * kMixRows;
  const int rows = min(kMixRows, tile.z - sub);
  if (rows <= 0) {
    pdl_wait();
    return;
  }
  const int t0 = tile.y + sub, pos0 = tile.w + sub;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q2 = (lane & 3) * 2;
  const int in8 = lane & 7, second = (lane >> 3) & 1, third = lane >> 4;
  const uint32_t base = smem_address(mix_smem);
  const int dim = a.dim, vdim = a.vdim, heads = a.heads, per = heads / a.kv_heads;
  const int last_pos = pos0 + rows - 1;
  const int lowest = a.window > 0 ? max(0, pos0 - a.window + 1) : 0;
  const int first_tile = lowest / kMixKeys, end_tile = last_pos / kMixKeys + 1;
  const int* table = a.block_table + (long long)tile.x * a.table_width;
  bool bad_page = false;
  auto find_places = [&](int t) {
    if (threadIdx.x < kMixKeys) {
      const int j = t * kMixKeys + threadIdx.x;
      int row = -1;
      if (j >= lowest && j <= last_pos) {
        const int logical = j / a.page_size, page = table[logical];
        if (page < 0 || page >= a.num_pages) bad_page = true;
        else row = page * a.kv_heads * a.page_size + (j - logical * a.page_size);
      }
      places[t & 1][threadIdx.x] = row;
    }
  };
  find_places(first_tile);

  // ---- q', summed in registers in the layout of a product's first operand.  All heads' queries of these rows come through
  // shared memory, as many heads at a time as it holds; rows of an odd number of 16-byte pieces.
  const int q_pitch = dim * 2 + 16, at_once = kMixSmem<VALUE> / (kMixRows * q_pitch);
  float mixed[kSteps][8];
#pragma unroll
  for (int kk = 0; kk < kSteps; ++kk)
#pragma unroll
    for (int e = 0; e < 8; ++e) mixed[kk][e] = 0.f;
  float slope = 0.f;
  pdl_wait();
  for (int g0 = 0; g0 < heads; g0 += at_once) {
    const int count = min(at_once, heads - g0), pieces = dim / 8;
    if (g0) __syncthreads();
    for (int i = threadIdx.x; i < kMixRows * count * pieces; i += kMixThreads) {
      const int r = i / (count * pieces), rest = i - r * (count * pieces), head = rest / pieces, piece = rest - head * pieces;
      const bool there = r < rows;
      cp_async16(base + (head * kMixRows + r) * q_pitch + piece * 16,
                 a.q + ((long long)(t0 + (there ? r : 0)) * heads + g0 + head) * dim + piece * 8, there ? 16 : 0);
    }
    cp_async_commit_group();
    cp_async_wait_groups<0>();
    __syncthreads();
    for (int u = 0; u < count; ++u) {
      const int other = g0 + u, c = other / per;
      const float w = a.talk ? a.talk[h * heads + other] : (other == h ? 1.f : 0.f);
      if (a.slopes) slope = fmaf(w, a.slopes[other], slope);
#pragma unroll
      for (int kk = 0; kk < kSteps; ++kk) {
        const int d = 16 * kk - c * dim;               // this head's 16 elements, if they are
        if (d < 0 || d >= dim) continue;
        uint32_t f[4];
        ldsm_x4(f, base + (u * kMixRows + 16 * warp + in8 + 8 * second) * q_pitch + (d / 8 + third) * 16);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          mixed[kk][2 * e] = fmaf(w, low_bf16(f[e]), mixed[kk][2 * e]);
          mixed[kk][2 * e + 1] = fmaf(w, high_bf16(f[e]), mixed[kk][2 * e + 1]);
        }
      }
    }
  }
  slope *= 1.4426950408889634f;
  __syncthreads();                                     // everyone has used the queries: their place takes the parts of q'
#pragma unroll
  for (int kk = 0; kk < kSteps; ++kk)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint32_t part[3];
      split3(mixed[kk][2 * e] * a.scale_log2, mixed[kk][2 * e + 1] * a.scale_log2, part);
      const uint32_t at = base + swizzled(16 * warp + g + 8 * (e & 1), 2 * kk + (e >> 1), kKeyPitch) + q2 * 2;
#pragma unroll
      for (int p = 0; p < 3; ++p) sts_u32(at + p * kQPart, part[p]);
    }
  __syncwarp();                                        // a warp's rows are its own

  // 64 rows: a thread has one 16-byte piece of every 128-byte line of four rows
  const int r0 = threadIdx.x >> 3, piece = threadIdx.x & 7;
  auto bring = [&](uint32_t at, auto lines_tag, const __nv_bfloat16* cache, int size, int first_head, int width, int t) {
    constexpr int kLines = decltype(lines_tag)::value, kPitch = 128 * kLines;
    int row[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) row[u] = places[t & 1][r0 + 16 * u];
#pragma unroll
    for (int line = 0; line < kLines; ++line) {
      const int e = 64 * line + 8 * piece, c = e / size;
      const bool inside = e < width;
      const __nv_bfloat16* from = cache + (long long)(first_head + c) * a.page_size * size + (e - c * size);
      const uint32_t to = at + r0 * kPitch + 128 * line + ((piece ^ r0) & 7) * 16;       // rows 16 apart exchange alike
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool there = inside && row[u] >= 0;
        cp_async16(to + u * 16 * kPitch, there ? from + (long long)row[u] * size : cache, there ? 16 : 0);
      }
    }
    cp_async_commit_group();
  };
  auto bring_keys = [&](int t) {
    bring(base + kK, std::integral_constant<int, kMixKeySize / 64>{}, a.k_cache, dim, 0, a.kv_heads * dim, t);
  };
  auto bring_values = [&](int t) {
    bring(base + kV, std::integral_constant<int, VALUE / 64>{}, a.v_cache, vdim, h / per, vdim, t);
  };
  bring_keys(first_tile);
  bring_values(first_tile);

  float O[VALUE / 8][4], m[2], l[2];
#pragma unroll
  for (int j = 0; j < VALUE / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) O[j][e] = 0.f;
  // the sink is the first term of every row's sum (counted once, by the first of the row's four lanes)
  m[0] = m[1] = a.sink ? a.sink[h] * 1.4426950408889634f : -INFINITY;
  l[0] = l[1] = a.sink && q2 == 0 ? 1.f : 0.f;
  const int warp_first = pos0 + 16 * warp, warp_last = warp_first + 15;

  for (int t = first_tile; t < end_tile; ++t) {
    const int j0 = t * kMixKeys;
    // a warp none of whose rows sees a key of the tile sits the products out
    const bool seen = j0 <= warp_last && (a.window <= 0 || j0 + kMixKeys - 1 > warp_first - a.window);
    if (t + 1 < end_tile) find_places(t + 1);
    cp_async_wait_groups<1>();                         // the keys are there
    __syncthreads();
    float S[8][4];
    if (seen) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j][e] = 0.f;
#pragma unroll 2
      for (int kk = 0; kk < kSteps; ++kk) {
        // as mma_parts does it, the eight column tiles side by side: small parts first, the sum of 16 elements added
        // to the running one by a rounded addition
        uint32_t qf[3][4], kf[4][4];
        float sum[8][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          ldsm_x4(kf[j], base + kK + swizzled(16 * j + in8 + 8 * third, 2 * kk + second, kKeyPitch));
#pragma unroll
        for (int p = 2; p >= 0; --p) {
          ldsm_x4(qf[p], base + p * kQPart + swizzled(16 * warp + in8 + 8 * second, 2 * kk + third, kKeyPitch));
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (p == 2) mma_bf16_16816_zero(sum[j], qf[p], kf[j >> 1][2 * (j & 1)], kf[j >> 1][2 * (j & 1) + 1]);
            else mma_bf16_16816(sum[j], qf[p], kf[j >> 1][2 * (j & 1)], kf[j >> 1][2 * (j & 1) + 1]);
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[j][e] += sum[j][e];
      }
    }
    __syncthreads();                                   // the keys are used up
    if (t + 1 < end_tile) bring_keys(t + 1);
    else cp_async_commit_group();                      // an empty group: the values are always the second youngest
    if (seen) {
      const bool masks = j0 + kMixKeys - 1 > warp_first || (a.window > 0 && j0 <= warp_last - a.window);
#pragma unroll
      for (int half = 0; half < 2; ++half) {           // rows g and g + 8 of the 16
        const int pos = warp_first + g + 8 * half;
        float top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int key = j0 + 8 * j + q2 + e;
            float z = S[j][2 * half + e] - slope * (float)(pos - key);
            if (masks) z = (key <= pos && (a.window <= 0 || key > pos - a.window)) ? z : -INFINITY;
            S[j][2 * half + e] = z;
            top = fmaxf(top, z);
          }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float to = fmaxf(m[half], top);
        const float shift = to == -INFINITY ? 0.f : to;
        const float factor = exp2f(m[half] - shift);   // nothing seen so far: zero
        m[half] = to;
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float w = exp2f(S[j][2 * half + e] - shift);
            S[j][2 * half + e] = w;
            sum += w;
          }
        l[half] = l[half] * factor + sum;              // this lane's share; the row's lanes are added at the end
        if (__any_sync(0xffffffffu, factor != 1.f)) {
#pragma unroll
          for (int j = 0; j < VALUE / 8; ++j) {
            O[j][2 * half] *= factor;
            O[j][2 * half + 1] *= factor;
          }
        }
      }
    }
    cp_async_wait_groups<1>();                         // the values are there
    __syncthreads();
    if (seen) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {                 // the weights are the first operand as they lie in registers
        uint32_t P[PARTS][4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          split_weights<PARTS>(S[2 * kk + (e >> 1)][2 * (e & 1)], S[2 * kk + (e >> 1)][2 * (e & 1) + 1], P, e);
        if constexpr (PARTS == 3) {
#pragma unroll
          for (int j = 0; j < VALUE / 16; j += 2) {
            uint32_t vf[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u)
              ldsm_x4_trans(vf[u], base + kV + swizzled(16 * kk + in8 + 8 * second, 2 * (j + u) + third, kValuePitch));
            add_weighted(O + 2 * j, P, vf);
          }
        } else {
#pragma unroll
          for (int j0v = 0; j0v < VALUE / 16; j0v += 4) {
            uint32_t vf[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
              ldsm_x4_trans(vf[j], base + kV + swizzled(16 * kk + in8 + 8 * second, 2 * (j0v + j) + third, kValuePitch));
#pragma unroll
            for (int p = PARTS - 1; p >= 0; --p)
#pragma unroll
              for (int j = 0; j < 8; ++j)
                mma_bf16_16816(O[2 * j0v + j], P[p], vf[j >> 1][2 * (j & 1)], vf[j >> 1][2 * (j & 1) + 1]);
          }
        }
      }
    }
    __syncthreads();                                   // the values are used up
    if (t + 1 < end_tile) bring_values(t + 1);
    else cp_async_commit_group();
  }
  cp_async_wait_groups<0>();
  if (bad_page) atomicOr(a.status, kStatusBadPage);

#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int r = 16 * warp + g + 8 * half;
    float sum = l[half];
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (r >= rows) continue;
    const float factor = sum > 0.f ? a.out_scale / sum : 0.f;
    __nv_bfloat16* out = a.out + ((long long)(t0 + r) * heads + h) * vdim;
#pragma unroll
    for (int j = 0; j < VALUE / 8; ++j) {
      const int column = 8 * j + q2;
      if (column < vdim)
        *reinterpret_cast<uint32_t*>(out + column) = pack_pair(O[j][2 * half] * factor, O[j][2 * half + 1] * factor);
    }
  }
}

// The same for requests that bring one token (decoding), up to 16 heads: a product's 16 rows are the token's heads, so a key
// or value row is read once for all of them, and its columns are all key heads end to end, then all value heads (a row uses
// those of its own head).  A CTA has a share of the token's keys, a warp 32 keys at a time of its own, brought by the warp
// alone: no barrier between the first key and the last.  What the warps found (maximum, sum, values) meets in shared memory,
// what the CTAs of a token found in the join below.
//
// Bound by the latencies of a CTA's few chunks.  Measured (B200): 64 tokens behind 2,048, 14 heads of 64 on 2, four CTAs a
// token: 68 -> 25 us (the FMA kernel of attention_mixed_tiled.cu; 23 with weights of two parts), the join 2.8 either way.
constexpr int kSingleChunk = 32, kSingleHeads = 16, kSinglePitch = 256;
constexpr int kSingleQ = 3 * kSingleHeads * kSinglePitch, kSingleWarp = 2 * kSingleChunk * kSinglePitch;
constexpr int kSingleSmem = kSingleQ + 4 * kSingleWarp, kSingleOPitch = 136;

struct SingleArgs {
  MixArgs m;
  const int* seq_of_token; const int* positions;
  const int* tokens;                 // token indices; null: token = block
  int splits, num_tokens;
  float* part_acc;                   // [splits, tokens, heads * vdim]
  float* part_ml;                    // [splits, tokens, heads, 2]: maximum (of scores in powers of two), sum
};

__global__ void __launch_bounds__(kMixThreads, 2)
mixed_single_attention_kernel(const __grid_constant__ SingleArgs s) {
  extern __shared__ __align__(128) unsigned char mix_smem[];
  __shared__ float mixing[kSingleHeads * kSingleHeads], slopes[kSingleHeads], warp_m[4][kSingleHeads], warp_l[4][kSingleHeads];
  const MixArgs& a = s.m;
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q2 = (lane & 3) * 2;
  const int in8 = lane & 7, second = (lane >> 3) & 1, third = lane >> 4;
  const uint32_t base = smem_address(mix_smem), keys_at = base + kSingleQ + warp * kSingleWarp;
  const uint32_t values_at = keys_at + kSingleChunk * kSinglePitch;
  const int dim = a.dim, vdim = a.vdim, heads = a.heads, per = heads / a.kv_heads;
  const int key_width = a.kv_heads * dim, value_width = a.kv_heads * vdim;
  const int t = s.tokens ? s.tokens[blockIdx.x] : (int)blockIdx.x;
  const int pos = s.positions[t];
  const int* table = a.block_table + (long long)s.seq_of_token[t] * a.table_width;
  const int lowest = a.window > 0 ? max(0, pos - a.window + 1) : 0;
  const int chunks = pos / kSingleChunk + 1 - lowest / kSingleChunk, share = (chunks + s.splits - 1) / s.splits;
  const int begin = lowest / kSingleChunk + (int)blockIdx.y * share, end = min(begin + share, pos / kSingleChunk + 1);
  bool bad_page = false;
  auto find = [&](int chunk) {       // of this lane's key: the page's first row of head 0 + slot in it, -1: none
    const int j = chunk * kSingleChunk + lane;
    if (chunk >= end || j < lowest || j > pos) return -1;
    const int logical = j / a.page_size, page = table[logical];
    if (page < 0 || page >= a.num_pages) {
      bad_page = true;
      return -1;
    }
    return page * a.kv_heads * a.page_size + (j - logical * a.page_size);
  };
  int chunk = begin + warp, row = find(chunk);
  const int piece = lane & 15, half_row = lane >> 4;
  auto bring = [&](uint32_t at, const __nv_bfloat16* cache, int size, int width, int rows) {
    const int e = 8 * piece, c = e / size;
    const __nv_bfloat16* from = cache + (long long)c * a.page_size * size + (e - c * size);
#pragma unroll
    for (int i = 0; i < kSingleChunk / 2; ++i) {
      const int key = 2 * i + half_row, place = __shfl_sync(0xffffffffu, rows, key);
      const bool there = e < width && place >= 0;
      cp_async16(at + swizzled(key, piece, kSinglePitch), there ? from + (long long)place * size : cache, there ? 16 : 0);
    }
  };
  // A chunk of earlier steps' keys alone (this step writes the last position's) is asked for before the wait, and what of
  // the mixing does not depend on the queries is made there too: the heads' weights in shared memory, where they do
  // not come from L2 one behind the other between the products of q', and the mixed slopes.  (With the token input's rows
  // and lines in stream_tail_tokens_kernel: four layers of 14 heads, 64 users behind 2,048, 516 -> 473 us a step.)
  const bool early = chunk < end && (chunk + 1) * kSingleChunk <= pos;
  auto bring_first = [&] {
    bring(keys_at, a.k_cache, dim, key_width, row);
    cp_async_commit_group();
    bring(values_at, a.v_cache, vdim, value_width, row);
    cp_async_commit_group();
  };
  if (early) bring_first();
  for (int i = threadIdx.x; i < kSingleHeads * kSingleHeads; i += kMixThreads) {
    const int h = i / kSingleHeads, other = i - h * kSingleHeads;
    mixing[i] = h < heads && other < heads ? (a.talk ? a.talk[h * heads + other] : (other == h ? 1.f : 0.f)) : 0.f;
  }
  __syncthreads();
  if (threadIdx.x < kSingleHeads) {
    float slope = 0.f;
    if (a.slopes)
      for (int other = 0; other < heads; ++other) slope = fmaf(mixing[threadIdx.x * kSingleHeads + other], a.slopes[other], slope);
    slopes[threadIdx.x] = slope * 1.4426950408889634f;
  }
  pdl_wait();
  if (!early) {
    if (chunk < end) {
      bring_first();
    } else {
      cp_async_commit_group();
      cp_async_commit_group();
    }
  }

  // ---- q': a thread has two neighbouring columns of every other head
  {
    const int e = 2 * ((int)threadIdx.x & 63), c = e / dim;
    float qx[kSingleHeads], qy[kSingleHeads];
#pragma unroll
    for (int u = 0; u < kSingleHeads; ++u) {
      const bool there = e < key_width && u < per;
      const uint32_t pair = there ? *reinterpret_cast<const uint32_t*>(a.q + ((long long)t * heads + c * per + u) * dim + e - c * dim) : 0u;
      qx[u] = low_bf16(pair);
      qy[u] = high_bf16(pair);
    }
    for (int h = threadIdx.x >> 6; h < kSingleHeads; h += 2) {
      float x = 0.f, y = 0.f;
      if (h < heads && e < key_width) {
#pragma unroll
        for (int u = 0; u < kSingleHeads; ++u) {
          if (u >= per) continue;
          const float w = mixing[h * kSingleHeads + c * per + u];
          x = fmaf(w, qx[u], x);
          y = fmaf(w, qy[u], y);
        }
      }
      uint32_t part[3];
      split3(x * a.scale_log2, y * a.scale_log2, part);
#pragma unroll
      for (int p = 0; p < 3; ++p)
        sts_u32(base + p * kSingleHeads * kSinglePitch + swizzled(h, e / 8, kSinglePitch) + (e & 7) * 2, part[p]);
    }
  }
  __syncthreads();
  const float slope[2] = {slopes[g], slopes[g + 8]};

  float O[16][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 16; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) O[j][e] = 0.f;
  for (; chunk < end; chunk += 4) {
    const int j0 = chunk * kSingleChunk;
    row = find(chunk + 4);
    cp_async_wait_groups<1>();                         // the keys are there
    __syncwarp();
    float S[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = 0.f;
#pragma unroll 2
    for (int kk = 0; kk < kMixKeySize / 16; ++kk) {
      if (16 * kk >= key_width) break;
      uint32_t qf[3][4], kf[2][4];
      float sum[4][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
        ldsm_x4(kf[j], keys_at + swizzled(16 * j + in8 + 8 * third, 2 * kk + second, kSinglePitch));
#pragma unroll
      for (int p = 2; p >= 0; --p) {
        ldsm_x4(qf[p], base + p * kSingleHeads * kSinglePitch + swizzled(in8 + 8 * second, 2 * kk + third, kSinglePitch));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (p == 2) mma_bf16_16816_zero(sum[j], qf[p], kf[j >> 1][2 * (j & 1)], kf[j >> 1][2 * (j & 1) + 1]);
          else mma_bf16_16816(sum[j], qf[p], kf[j >> 1][2 * (j & 1)], kf[j >> 1][2 * (j & 1) + 1]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j][e] += sum[j][e];
    }
    __syncwarp();                                      // the keys are used up
    if (chunk + 4 < end) bring(keys_at, a.k_cache, dim, key_width, row);
    cp_async_commit_group();                           // perhaps an empty group: the values are always the second youngest
#pragma unroll
    for (int half = 0; half < 2; ++half) {             // heads g and g + 8
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int key = j0 + 8 * j + q2 + e;
          const float z = S[j][2 * half + e] - slope[half] * (float)(pos - key);
          S[j][2 * half + e] = key >= lowest && key <= pos ? z : -INFINITY;
          top = fmaxf(top, S[j][2 * half + e]);
        }
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
      const float to = fmaxf(m[half], top);
      const float shift = to == -INFINITY ? 0.f : to;
      const float factor = exp2f(m[half] - shift);     // nothing seen so far: zero
      m[half] = to;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float w = exp2f(S[j][2 * half + e] - shift);
          S[j][2 * half + e] = w;
          sum += w;
        }
      l[half] = l[half] * factor + sum;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        O[j][2 * half] *= factor;
        O[j][2 * half + 1] *= factor;
      }
    }
    cp_async_wait_groups<1>();                         // the values are there
    __syncwarp();
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      uint32_t P[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        split_weights<3>(S[2 * kk + (e >> 1)][2 * (e & 1)], S[2 * kk + (e >> 1)][2 * (e & 1) + 1], P, e);
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        if (16 * j >= value_width) break;              // the last pair may reach into columns of zeros
        uint32_t vf[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          ldsm_x4_trans(vf[u], values_at + swizzled(16 * kk + in8 + 8 * second, 2 * (j + u) + third, kSinglePitch));
        add_weighted(O + 2 * j, P, vf);
      }
    }
    __syncwarp();                                      // the values are used up
    if (chunk + 4 < end) bring(values_at, a.v_cache, vdim, value_width, row);
    cp_async_commit_group();
  }
  cp_async_wait_groups<0>();
  if (bad_page) atomicOr(a.status, kStatusBadPage);
  __syncthreads();                                     // everyone is done with the tiles: their place takes the warps' results
  float* found = reinterpret_cast<float*>(mix_smem + kSingleQ);       // [warp, head, value column]
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int h = g + 8 * half;
    float sum = l[half];
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (q2 == 0) {
      warp_m[warp][h] = m[half];
      warp_l[warp][h] = sum;
    }
    float* to = found + (warp * kSingleHeads + h) * kSingleOPitch + q2;
#pragma unroll
    for (int j = 0; j < 16; ++j) *reinterpret_cast<float2*>(to + 8 * j) = make_float2(O[j][2 * half], O[j][2 * half + 1]);
  }
  __syncthreads();
  const int outs = heads * vdim;
  const size_t part = ((size_t)blockIdx.y * s.num_tokens + t);
  for (int o = threadIdx.x; o < outs; o += kMixThreads) {
    const int h = o / vdim, d = o - h * vdim, column = (h / per) * vdim + d;
    const bool whole = s.splits == 1;
    float best = whole && a.sink ? a.sink[h] * 1.4426950408889634f : -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) best = fmaxf(best, warp_m[w][h]);
    float sum = whole && a.sink ? exp2f(a.sink[h] * 1.4426950408889634f - best) : 0.f, value = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float factor = warp_m[w][h] == -INFINITY ? 0.f : exp2f(warp_m[w][h] - best);
      sum = fmaf(warp_l[w][h], factor, sum);
      value = fmaf(found[(w * kSingleHeads + h) * kSingleOPitch + column], factor, value);
    }
    if (whole) {
      a.out[(size_t)t * outs + o] = __float2bfloat16_rn(sum > 0.f ? value / sum * a.out_scale : 0.f);
    } else {
      s.part_acc[part * outs + o] = value;
      if (d == 0) *reinterpret_cast<float2*>(s.part_ml + (part * heads + h) * 2) = make_float2(best, sum);
    }
  }
}

__global__ void __launch_bounds__(kMixThreads) mixed_single_join_kernel(const __grid_constant__ SingleArgs s) {
  const MixArgs& a = s.m;
  pdl_launch_dependents();
  const int outs = a.heads * a.vdim, o = (int)blockIdx.y * kMixThreads + (int)threadIdx.x;
  const int t = s.tokens ? s.tokens[blockIdx.x] : (int)blockIdx.x;
  pdl_wait();
  if (o >= outs) return;
  const int h = o / a.vdim;
  const size_t ml_step = (size_t)s.num_tokens * a.heads, acc_step = (size_t)s.num_tokens * outs;
  const float2* ml = reinterpret_cast<const float2*>(s.part_ml) + (size_t)t * a.heads + h;
  const float* acc = s.part_acc + (size_t)t * outs + o;
  constexpr int kBatch = 8;                            // loads in flight before they are used
  float best = a.sink ? a.sink[h] * 1.4426950408889634f : -INFINITY;
  float sum = a.sink ? 1.f : 0.f, value = 0.f;
  for (int s0 = 0; s0 < s.splits; s0 += kBatch) {
    float2 of[kBatch];
    float v[kBatch];
    float to = best;
#pragma unroll
    for (int e = 0; e < kBatch; ++e) {
      const bool there = s0 + e < s.splits;
      of[e] = there ? ml[(s0 + e) * ml_step] : make_float2(-INFINITY, 0.f);
      v[e] = there ? acc[(s0 + e) * acc_step] : 0.f;
      to = fmaxf(to, of[e].x);
    }
    const float factor = best == -INFINITY ? 0.f : exp2f(best - to);
    sum *= factor;
    value *= factor;
    best = to;
#pragma unroll
    for (int e = 0; e < kBatch; ++e) {
      const float w = of[e].x == -INFINITY ? 0.f : exp2f(of[e].x - best);
      sum = fmaf(of[e].y, w, sum);
      value = fmaf(v[e], w, value);
    }
  }
  a.out[(size_t)t * outs + o] = __float2bfloat16_rn(sum > 0.f ? value / sum * a.out_scale : 0.f);
}

template <int VALUE, int PARTS>
static cudaError_t launch_mixed_prompt(const MixArgs& a, int num_tiles, cudaStream_t stream) {
  auto kernel = mixed_prompt_attention_kernel<VALUE, PARTS>;
  constexpr int kBytes = kMixSmem<VALUE>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return e;
  return launch_pdl(kernel, dim3(2 * num_tiles * a.heads), dim3(kMixThreads), kBytes, stream, a);
}

}  // namespace einf

using namespace einf;

// The portions of up to 128 tokens that `tiles` lists; `wave`: multiprocessors of the device.
extern "C" int einf_mixed_prompt_attention(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                                           int table_width, const int* tiles, int num_tiles, void* out, int heads, int kv_heads,
                                           int dim, int vdim, int page_size, int num_pages, float scale, int window,
                                           const float* slopes, const float* talk, const float* sink, float out_scale, int wave,
                                           int* status, cudaStream_t stream) {
  if (num_tiles == 0) return 0;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || dim <= 0 || dim % 16 || kv_heads * dim > kMixKeySize || vdim <= 0 ||
      vdim % 8 || vdim > 128 || 2ll * num_tiles * heads > 0x7fffffff || wave <= 0 ||
      (long long)num_pages * kv_heads * page_size > 0x7fffffff ||
      (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)tiles) & 15) || ((uintptr_t)out & 3))
    return (int)cudaErrorInvalidValue;
  MixArgs a;
  a.q = (const __nv_bfloat16*)q;
  a.k_cache = (const __nv_bfloat16*)k_cache; a.v_cache = (const __nv_bfloat16*)v_cache;
  a.block_table = block_table; a.table_width = table_width;
  a.tiles = (const int4*)tiles; a.out = (__nv_bfloat16*)out;
  a.slopes = slopes; a.talk = talk; a.sink = sink; a.status = status;
  a.heads = heads; a.kv_heads = kv_heads; a.dim = dim; a.vdim = vdim; a.page_size = page_size; a.num_pages = num_pages;
  a.window = window; a.wave = wave;
  a.scale_log2 = scale * 1.4426950408889634f; a.out_scale = out_scale;
  if (heads <= 16)
    return (int)(vdim <= 64 ? launch_mixed_prompt<64, 2>(a, num_tiles, stream) : launch_mixed_prompt<128, 2>(a, num_tiles, stream));
  return (int)(vdim <= 64 ? launch_mixed_prompt<64, 3>(a, num_tiles, stream) : launch_mixed_prompt<128, 3>(a, num_tiles, stream));
}

// One token each of `num_items` requests (`items`: token indices, null: tokens 0 .. num_items - 1); `splits` CTAs share a
// token's keys and, above one, need part_acc [splits, num_tokens, heads * vdim] and part_ml [splits, num_tokens, heads, 2].
extern "C" int einf_mixed_single_attention(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                                           int table_width, const int* seq_of_token, const int* positions, const int* items,
                                           int num_items, void* out, int num_tokens, int heads, int kv_heads, int dim, int vdim,
                                           int page_size, int num_pages, float scale, int window, const float* slopes,
                                           const float* talk, const float* sink, float out_scale, int splits, float* part_acc,
                                           float* part_ml, int* status, cudaStream_t stream) {
  if (num_items == 0) return 0;
  if (heads <= 0 || heads > kSingleHeads || kv_heads <= 0 || heads % kv_heads || dim <= 0 || dim % 8 ||
      kv_heads * dim > kMixKeySize || vdim <= 0 || vdim % 8 || kv_heads * vdim > 128 || splits < 1 || splits > 65535 ||
      (splits > 1 && (!part_acc || !part_ml)) || (long long)num_pages * kv_heads * page_size > 0x7fffffff ||
      (((uintptr_t)k_cache | (uintptr_t)v_cache) & 15) || ((uintptr_t)q & 3) || ((uintptr_t)part_ml & 7))
    return (int)cudaErrorInvalidValue;
  SingleArgs s;
  MixArgs& a = s.m;
  a.q = (const __nv_bfloat16*)q;
  a.k_cache = (const __nv_bfloat16*)k_cache; a.v_cache = (const __nv_bfloat16*)v_cache;
  a.block_table = block_table; a.table_width = table_width; a.tiles = nullptr; a.out = (__nv_bfloat16*)out;
  a.slopes = slopes; a.talk = talk; a.sink = sink; a.status = status;
  a.heads = heads; a.kv_heads = kv_heads; a.dim = dim; a.vdim = vdim; a.page_size = page_size; a.num_pages = num_pages;
  a.window = window; a.wave = 0;
  a.scale_log2 = scale * 1.4426950408889634f; a.out_scale = out_scale;
  s.seq_of_token = seq_of_token; s.positions = positions; s.tokens = items;
  s.splits = splits; s.num_tokens = num_tokens; s.part_acc = part_acc; s.part_ml = part_ml;
  cudaError_t e = cudaFuncSetAttribute(mixed_single_attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSingleSmem);
  if (e != cudaSuccess) return (int)e;
  e = launch_pdl(mixed_single_attention_kernel, dim3(num_items, splits), dim3(kMixThreads), kSingleSmem, stream, s);
  if (e != cudaSuccess || splits == 1) return (int)e;
  return (int)launch_pdl(mixed_single_join_kernel, dim3(num_items, (heads * vdim + kMixThreads - 1) / kMixThreads),
                         dim3(kMixThreads), 0, stream, s);
}
