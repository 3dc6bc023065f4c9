// The linear recurrence of recurrence.cu for prompts, 64 tokens at a time on the tensor cores.
//
//   S <- a_t S + k_t (s_t v_t)^T,      y_t = S^T q_t + skip_h v_t
//
// Over a chunk of tokens that starts from the state S0 the same sums read, with D[t, s] the product of the decays a of
// the tokens s + 1 .. t and d0[t] the product of all decays up to t,
//   y_t = d0[t] (S0^T q_t) + sum_{s <= t} (q_t . k_s) D[t, s] s_s v_s,
//   S1  = d0[last] S0 + sum_s k_s (D[last, s] s_s v_s)^T,
// four matrix products in the place of one dependent step per token.  The token-by-token kernel is bound by its 32-bit FMA
// (4 dim vdim per token, once and a half, at 70 TFLOP/s over the GPU) and by the chain of its steps; these products run at
// the rate of mma.sync.  Nothing is rounded below 32 bits: q, k and v as the caller stores them are bfloat16
// already and enter as they are; a 32-bit operand (the state, the weights (q . k) D s, the weighted values, and
// q, k, v behind a SiLU) enters as three bfloat16 parts (mma_sync.cuh), with three products against a
// bfloat16 operand and six against another 32-bit one; all sums are 32-bit.  The products of decays are multiplied out,
// never divided or taken from logarithms, so that a decay of zero stays one: inside a tile of 16 tokens
// token after token, across tiles as (tokens of t's tile up to t) (whole tiles between) (tokens of s's tile behind s).
// They are multiplied in 64 bits and rounded once: with one decay for all tokens of a head the roundings of a 32-bit
// product of 64 of them are the same in every chunk and add up over a long memory (measured: a state 1.4e-6 off
// where the token-by-token kernel, whose roundings differ from step to step, is 2.4e-7 off, and this one 8e-8).
//
// A CTA has one head, a run of columns of its state and one segment of a portion, eight warps: warp w has the 16 tokens
// w % 4 of the chunk's 64 in the first three products and a quarter of the state's rows in the last, of half the columns.
// Long portions are cut into segments as in recurrence.cu: a pass over all segments from a zero state, a walk that
// leaves every segment's start state (here as three bfloat16 parts, which the last pass brings straight into shared
// memory), the emitting pass.  Only portions of min_len tokens and more are taken (the others are recurrence.cu's).  Their
// segments are numbered q_start[r] / segment_len + (such portions before r) + (segment of the portion), which leaves no two
// portions a common number and stays below tokens / segment_len + portions, however long the longest of them: users
// that decode beside a prompt cost neither segments nor CTAs.
//
// Measured (B200, bfloat16, the three launches of a call, token-by-token kernel before): lightning attention, 14 heads of
// 64 x 64, prompts of 4,096 and 1,000 tokens 222 -> 105 us; Mamba-2, 24 heads of 128 x 64, 2,048 tokens 242 -> 70 us; matrix
// memory, 6 heads of 128 x 260, prompts of 2,048 and 500 tokens 332 -> 93 us (7 heads of 64 x 132, 1,500 and 301: 121 -> 37
// us).  The error against 64 bits is no larger: 0.9, 0.9 and 1.1e-7 of y's norm (before: 1.7, 1.0 and 1.4e-7).  What bounds
// it now are its instructions beside the products (taking values apart into parts, rounded additions) and, at two CTAs
// an SM, the latency of its loads.
//
// The weights beyond the diagonal of a tile of 16 tokens are zeros, and zero times a value that is not finite is NaN: such
// values leave the product of their own tile and are added one by one to the tokens they belong to, so that none reaches a
// token before its own.
#include <type_traits>

#include "mma_sync.cuh"

namespace einf {

constexpr int kChunk = 64;             // tokens of a chunk
constexpr int kChunkThreads = 256;
constexpr int kDiagonalPitch = 24;     // floats of a row of a 16 x 16 tile of D: a fragment's 8-byte reads meet no bank twice

struct ChunkArgs {
  const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v;
  long long q_stride, k_stride, v_stride;
  const float* head_decay; const float* token_decay; const float* token_scale; const float* skip;
  float* state; long long state_stride;
  const int* q_start; const int* state_slots;
  float* y;
  float* segment_state;             // [segments, heads, dim, vdim]: what a segment adds, from zero
  __nv_bfloat16* segment_start;     // [segments, heads, 3, dim, vdim]: the state it starts from, in parts
  float* segment_decay;             // [segments, heads]
  int num_slots, num_requests, heads, groups, dim, vdim, segment_len;
  int min_len;                      // tokens of the shortest portion that is taken (at least one)
  int wide;                         // operands with 16-byte rows (bits: q, k, v, the segments' start states)
};

// Which portion a CTA has: the request whose segments' numbers hold `number` or, with kByRank, the number-th that is taken
// (-1: none).  first_segment: the number of its first.  Every warp looks for itself, 32 requests at a time.
template <bool kByRank>
__device__ __forceinline__ int find_portion(const ChunkArgs& a, int number, int* first_segment) {
  const int lane = threadIdx.x & 31;
  int before = 0;                                // portions taken among the requests so far
#pragma unroll 4
  for (int base = 0; base < a.num_requests; base += 32) {
    const int i = base + lane;
    const int begin = i < a.num_requests ? a.q_start[i] : 0;
    const int count = i < a.num_requests ? a.q_start[i + 1] - begin : 0;
    const bool taken = count >= a.min_len;
    const uint32_t all = __ballot_sync(0xffffffffu, taken);
    const int rank = before + __popc(all & ((1u << lane) - 1u));
    const int first = begin / a.segment_len + rank;
    const bool mine = taken && (kByRank ? rank == number
                                        : first <= number && number < first + (count + a.segment_len - 1) / a.segment_len);
    const uint32_t found = __ballot_sync(0xffffffffu, mine);
    if (found) {
      const int at = __ffs(found) - 1;
      *first_segment = __shfl_sync(0xffffffffu, first, at);
      return base + at;
    }
    before += __popc(all);
  }
  return -1;
}

// SiLU with the quick division: two units in the last place at most (the division that rounds exactly is a third of this
// kernel's instructions where the inputs pass a SiLU; y and state stay closer to 64 bits than the token-by-token kernel's).
__device__ __forceinline__ float silu_quick(float z) { return __fdividef(z, 1.f + expf(-z)); }

// Shared memory of a CTA, in bytes from its start.  ROWS: rows of the state (filled up); NT: tiles of eight columns;
// with kAct the inputs are 32-bit values in three parts.  Rows of q and k (and of v and the state at 64 columns) are a
// power of two long, and their 16-byte pieces are exchanged by the row's last three bits; other rows are an odd
// number of pieces long.  Either way the eight rows of an ldmatrix meet no bank twice.
template <int ROWS, int NT, bool kAct, bool kEmit>
struct ChunkLayout {
  static constexpr int kInParts = kAct ? 3 : 1;
  static constexpr bool kSwizzled = NT == 8;
  static constexpr int kRowPitch = ROWS * 2;
  static constexpr int kColPitch = kSwizzled ? 128 : (NT | 1) * 16;
  static constexpr int kKey = 0;
  static constexpr int kKeyPart = kChunk * kRowPitch;
  static constexpr int kValue = kKey + kInParts * kKeyPart;      // in the first pass the weighted values take their place
  static constexpr int kValuePart = kChunk * kColPitch;
  static constexpr int kQuery = kValue + (kEmit ? kInParts : 3) * kValuePart;
  // the queries' place, and behind them that of the ten 16 x 16 tiles of q . k, which the halves of the warps exchange there
  static constexpr int kQueryBytes = kInParts * kKeyPart > 10 * 1024 ? kInParts * kKeyPart : 10 * 1024;
  static constexpr int kState = kQuery + (kEmit ? kQueryBytes : 0);
  static constexpr int kStatePart = ROWS * kColPitch;
  static constexpr int kDiagonal = kState + (kEmit ? 3 * kStatePart : 0);
  static constexpr int kVectors = kDiagonal + (kEmit ? kChunk * kDiagonalPitch * 4 : 0);   // 64 floats each
  static constexpr int kBytes = kVectors + 4 * kChunk * 4 + 4 * 8;
  // byte of a 16-byte piece in a row of v or of the state
  static __device__ __forceinline__ int column(int row, int piece) { return (kSwizzled ? (piece ^ (row & 7)) : piece) * 16; }
};

// `rows` rows of `width` elements to shared memory, zeros from row n on and beyond `width`: a thread has one place of a
// row, ELEMS elements long (4, or 8 where every row is 16-byte aligned), and steps through the rows.  CHUNKS: 16-byte
// pieces of a row in shared memory; kSwap: exchanged as above; kAct: through a SiLU into three parts.
template <int ELEMS, int CHUNKS, bool kSwap, bool kAct>
__device__ __forceinline__ void bring_rows(uint32_t at, int pitch, int part_bytes, const __nv_bfloat16* src, long long stride,
                                           int width, int n, int rows) {
  constexpr int kPieces = CHUNKS * 8 / ELEMS;              // in a row
  constexpr int kStep = kChunkThreads / kPieces;           // rows side by side over the threads
  const int row = threadIdx.x / kPieces, piece = threadIdx.x - row * kPieces;
  if (row >= kStep) return;
  const int chunk = piece * ELEMS / 8, in_chunk = (piece * ELEMS % 8) * 2;
  const bool inside = piece * ELEMS < width;
  const __nv_bfloat16* from = src + (long long)row * stride + piece * ELEMS;
  constexpr int kAtOnce = kAct ? 4 : 8;                    // loads in flight before the first is used
  for (int t = row; t < rows; t += kAtOnce * kStep) {
    if constexpr (!kAct) {
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u, from += kStep * stride) {
        const int tt = t + u * kStep;
        if (tt >= rows) break;
        const bool there = inside && tt < n;
        const uint32_t to = at + tt * pitch + (kSwap ? (chunk ^ (tt & 7)) : chunk) * 16 + in_chunk;
        if constexpr (ELEMS == 8) cp_async16(to, there ? from : src, there ? 16 : 0);
        else cp_async8(to, there ? from : src, there ? 8 : 0);
      }
    } else {
      uint32_t raw[kAtOnce][ELEMS / 2];
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u, from += kStep * stride) {
#pragma unroll
        for (int e = 0; e < ELEMS / 2; ++e) raw[u][e] = 0u;
        if (inside && t + u * kStep < n) {
          if constexpr (ELEMS == 8) {
            const uint4 v = *reinterpret_cast<const uint4*>(from);
            raw[u][0] = v.x; raw[u][1] = v.y; raw[u][2] = v.z; raw[u][3] = v.w;
          } else {
            const uint2 v = *reinterpret_cast<const uint2*>(from);
            raw[u][0] = v.x; raw[u][1] = v.y;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u) {
        const int tt = t + u * kStep;
        if (tt >= rows) break;
        const uint32_t to = at + tt * pitch + (kSwap ? (chunk ^ (tt & 7)) : chunk) * 16 + in_chunk;
#pragma unroll
        for (int e = 0; e < ELEMS / 2; e += 2) {
          uint32_t lo[3], hi[3];
          split3(silu_quick(low_bf16(raw[u][e])), silu_quick(high_bf16(raw[u][e])), lo);
          split3(silu_quick(low_bf16(raw[u][e + 1])), silu_quick(high_bf16(raw[u][e + 1])), hi);
#pragma unroll
          for (int p = 0; p < 3; ++p) sts_v2(to + p * part_bytes + e * 4, lo[p], hi[p]);
        }
      }
    }
  }
}
template <int CHUNKS, bool kSwap, bool kAct>
__device__ __forceinline__ void bring(bool wide, uint32_t at, int pitch, int part_bytes, const __nv_bfloat16* src,
                                      long long stride, int width, int n, int rows) {
  if (wide) bring_rows<8, CHUNKS, kSwap, kAct>(at, pitch, part_bytes, src, stride, width, n, rows);
  else bring_rows<4, CHUNKS, kSwap, kAct>(at, pitch, part_bytes, src, stride, width, n, rows);
}

// Two CTAs an SM, but for the emitting pass whose inputs in parts fill an SM's shared memory.
template <int ROWS, int NT, bool kAct, bool kEmit>
__global__ void __launch_bounds__(kChunkThreads, (ChunkLayout<ROWS, NT, kAct, kEmit>::kBytes > 113 * 1024 ? 1 : 2))
recurrence_chunk_kernel(const __grid_constant__ ChunkArgs a) {
  using L = ChunkLayout<ROWS, NT, kAct, kEmit>;
  extern __shared__ __align__(16) unsigned char chunk_smem[];
  pdl_launch_dependents();
  pdl_wait();
  constexpr int kColumns = NT * 8;
  constexpr int NH = NT / 2;                     // column tiles of a warp
  constexpr int kMT = ROWS / 64;                 // 16-row tiles of the state a warp owns
  constexpr int kIn = L::kInParts;
  constexpr int kUsed = kEmit ? kIn : 3;         // parts of the values when the state is updated
  const int lane = threadIdx.x & 31, tile = (threadIdx.x >> 5) & 3, half = threadIdx.x >> 7;
  const int g = lane >> 2, q2 = (lane & 3) * 2;  // a fragment's row and first column of this lane
  const int n0 = half * NH;                      // this warp's first column tile
  const int column0 = blockIdx.x * kColumns, head = blockIdx.y;
  int numbered;
  const int r = find_portion<false>(a, (int)blockIdx.z, &numbered);      // whose segment this CTA has
  if (r < 0) return;
  const int segment = (int)blockIdx.z - numbered;
  const int request_first = a.q_start[r], request_last = a.q_start[r + 1];
  const int slot = a.state_slots[r];
  const int count = request_last - request_first;
  const int num_segments = (count + a.segment_len - 1) / a.segment_len;
  if (!kEmit && num_segments <= 1) return;
  const int first = request_first + segment * a.segment_len;
  const int last = min(request_last, first + a.segment_len);
  const int dim = a.dim, vdim = a.vdim;
  const uint32_t base = smem_address(chunk_smem);
  float* vectors = reinterpret_cast<float*>(chunk_smem + L::kVectors);
  float* const decay = vectors;                  // a of the chunk's tokens
  float* const scale = vectors + kChunk;         // s
  float* const before = vectors + 2 * kChunk;    // product of the decays of t's tile up to t
  float* const behind = vectors + 3 * kChunk;    // product of the decays of s's tile behind s, times s_s
  double* const whole = reinterpret_cast<double*>(vectors + 4 * kChunk);      // product of the decays of a tile
  float* const diagonal = reinterpret_cast<float*>(chunk_smem + L::kDiagonal);

  // A portion of one segment starts from its slot and leaves its state there; of several, the walk did both.
  const long long in_head = (long long)head * dim * vdim;
  float* slot_state = nullptr;
  if (slot >= 0 && slot < a.num_slots) slot_state = a.state + (long long)slot * a.state_stride + in_head;
  const float* const start_state = kEmit && num_segments == 1 ? slot_state : nullptr;
  float* const end_state = !kEmit ? a.segment_state + (long long)blockIdx.z * a.heads * dim * vdim + in_head
                           : num_segments == 1 ? slot_state : nullptr;

  const int group = head / (a.heads / a.groups);
  const __nv_bfloat16* qg = a.q + (long long)group * dim;
  const __nv_bfloat16* kg = a.k + (long long)group * dim;
  const __nv_bfloat16* vg = a.v + (long long)head * vdim + column0;
  const float constant_decay = a.head_decay ? a.head_decay[head] : 1.f;
  const float skip = a.skip ? a.skip[head] : 0.f;
  const long long y_step = (long long)a.heads * vdim;

  if (kEmit && num_segments > 1) {
    const __nv_bfloat16* from = a.segment_start + 3 * ((long long)blockIdx.z * a.heads + head) * dim * vdim + column0;
#pragma unroll
    for (int p = 0; p < 3; ++p)
      bring<NT, L::kSwizzled, false>(a.wide & 8, base + L::kState + p * L::kStatePart, L::kColPitch, 0,
                                     from + (long long)p * dim * vdim, vdim, vdim - column0, dim, ROWS);
  } else if (kEmit) {
    constexpr int kQuads = kColumns / 4;         // 16-byte pieces of a row
#pragma unroll 4
    for (int i = threadIdx.x; i < ROWS * kQuads; i += kChunkThreads) {
      const int row = i / kQuads, quad = i - row * kQuads;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (start_state && row < dim && column0 + 4 * quad < vdim)
        v = *reinterpret_cast<const float4*>(start_state + (long long)row * vdim + column0 + 4 * quad);
      uint32_t lo[3], hi[3];
      split3(v.x, v.y, lo);
      split3(v.z, v.w, hi);
      const uint32_t at = base + L::kState + row * L::kColPitch + L::column(row, quad >> 1) + (quad & 1) * 8;
#pragma unroll
      for (int p = 0; p < 3; ++p) sts_v2(at + p * L::kStatePart, lo[p], hi[p]);
    }
  }

  // this warp's part of the state while it is updated: rows (tile * kMT + m) * 16 + g and + 8, columns 8 (n0 + j) + q2
  // and + 1
  float S[kMT][NH][4];
#pragma unroll
  for (int m = 0; m < kMT; ++m)
#pragma unroll
    for (int j = 0; j < NH; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[m][j][e] = 0.f;
  double decay_product = 1.;
  // rows of the fragment loads: eight each for lanes 0-7, 8-15, 16-23, 24-31
  const int in8 = lane & 7, second = (lane >> 3) & 1, third = lane >> 4;
  // two column tiles (the second operand) from 16 rows of v or of the state's parts; `at` is the buffer's start
  auto column_tiles = [&](uint32_t (&b0)[2], uint32_t (&b1)[2], int at, int row0, int tile0) {
    uint32_t f[4];
    const int row = row0 + in8 + 8 * second;
    ldsm_x4_trans(f, base + at + row * L::kColPitch + L::column(row, tile0 + third));
    b0[0] = f[0]; b0[1] = f[1]; b1[0] = f[2]; b1[1] = f[3];
  };
  auto column_tile = [&](uint32_t (&b)[2], int at, int row0, int tile0) {
    const int row = row0 + in8 + 8 * second;
    ldsm_x2_trans(b, base + at + row * L::kColPitch + L::column(row, tile0));
  };

  for (int t0 = first; t0 < last; t0 += kChunk) {
    const int n = min(kChunk, last - t0);
    const int tiles = (n + 15) >> 4;               // 16-token tiles with a token in them
    const bool more = t0 + kChunk < last;
    if (threadIdx.x < kChunk) {
      const int t = threadIdx.x;
      const bool there = t < n;
      decay[t] = there ? (a.token_decay ? a.token_decay[(long long)(t0 + t) * a.heads + head] : constant_decay) : 1.f;
      scale[t] = there ? (a.token_scale ? a.token_scale[(long long)(t0 + t) * a.heads + head] : 1.f) : 0.f;
    }
    bring<ROWS / 8, true, kAct>(a.wide & 2, base + L::kKey, L::kRowPitch, L::kKeyPart, kg + (long long)t0 * a.k_stride,
                                a.k_stride, dim, n, 16 * tiles);
    if (kEmit)
      bring<ROWS / 8, true, kAct>(a.wide & 1, base + L::kQuery, L::kRowPitch, L::kKeyPart, qg + (long long)t0 * a.q_stride,
                                  a.q_stride, dim, n, 16 * tiles);
    bring<NT, L::kSwizzled, kAct>(a.wide & 4, base + L::kValue, L::kColPitch, L::kValuePart, vg + (long long)t0 * a.v_stride,
                                  a.v_stride, vdim - column0, n, 16 * tiles);
    cp_async_commit_group();
    __syncthreads();
    if (threadIdx.x < kChunk) {                    // a column of its tile of D each
      const int s = threadIdx.x, in_tile = s & 15;
      const float* tile_decay = decay + (s & ~15);
      double d = scale[s];
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        if (t > in_tile) d *= (double)tile_decay[t];
        if (kEmit) diagonal[((s & ~15) + t) * kDiagonalPitch + in_tile] = t >= in_tile ? (float)d : 0.f;
      }
      behind[s] = (float)d;
    } else if (threadIdx.x < 2 * kChunk) {
      const int t = threadIdx.x - kChunk, in_tile = t & 15;
      const float* tile_decay = decay + (t & ~15);
      double d = 1.;
#pragma unroll
      for (int u = 0; u < 16; ++u)
        if (u <= in_tile) d *= (double)tile_decay[u];
      before[t] = (float)d;
      if (in_tile == 15) whole[t >> 4] = d;
    }
    cp_async_wait_groups<0>();
    __syncthreads();

    if constexpr (kEmit) {
      // (q_t . k_s) for this warp's 16 tokens t and the tokens s up to the last of them, every other tile of 16: the warp with
      // the same tokens and the other columns has the others (both made all of them before: of the last tokens' warps,
      // whose products are the CTA's longest chain, 96 products in place of 192 where both operands have three parts)
      const bool here = 16 * tile < n;
      float G[2][2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) G[i][j][e] = 0.f;
      const uint32_t q_at = base + L::kQuery + (16 * tile + in8 + 8 * second) * L::kRowPitch;
      const uint32_t k_at = base + L::kKey + (in8 + 8 * third + 16 * half) * L::kRowPitch;
      auto query = [&](uint32_t (&f)[kIn][4], int kk) {
#pragma unroll
        for (int p = 0; p < kIn; ++p) ldsm_x4(f[p], q_at + p * L::kKeyPart + ((2 * kk + third) ^ in8) * 16);
      };
      if (here) {
#pragma unroll 1
        for (int kk = 0; kk < ROWS / 16; ++kk) {
          uint32_t qf[kIn][4];
          query(qf, kk);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (half + 2 * i > tile) break;
            uint32_t k0[kIn][2], k1[kIn][2];
#pragma unroll
            for (int p = 0; p < kIn; ++p) {
              uint32_t f[4];
              ldsm_x4(f, k_at + p * L::kKeyPart + 32 * i * L::kRowPitch + ((2 * kk + second) ^ in8) * 16);
              k0[p][0] = f[0]; k0[p][1] = f[1]; k1[p][0] = f[2]; k1[p][1] = f[3];
            }
            mma_parts<kIn, kIn>(G[i][0], qf, k0);
            mma_parts<kIn, kIn>(G[i][1], qf, k1);
          }
        }
      }
      // what the chunk's start state gives: d0[t] S0^T q_t
      float Y[NH][4];
#pragma unroll
      for (int j = 0; j < NH; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) Y[j][e] = 0.f;
#pragma unroll 1
      for (int kk = 0; kk < (here ? ROWS / 16 : 0); ++kk) {
        uint32_t qf[kIn][4];
        query(qf, kk);
#pragma unroll
        for (int j = 0; j < NH / 2; ++j) {
          uint32_t s0[3][2], s1[3][2];
#pragma unroll
          for (int p = 0; p < 3; ++p) column_tiles(s0[p], s1[p], L::kState + p * L::kStatePart, 16 * kk, n0 + 2 * j);
          mma_parts<kIn, 3>(Y[2 * j], qf, s0);
          mma_parts<kIn, 3>(Y[2 * j + 1], qf, s1);
        }
        if constexpr (NH & 1) {
          uint32_t s0[3][2];
#pragma unroll
          for (int p = 0; p < 3; ++p) column_tile(s0[p], L::kState + p * L::kStatePart, 16 * kk, n0 + NH - 1);
          mma_parts<kIn, 3>(Y[NH - 1], qf, s0);
        }
      }
      __syncthreads();                             // everyone has read the queries
      auto exchanged = [&](int j, int e) {         // this lane's four of the tokens 16 j + 8 e on
        return chunk_smem + L::kQuery + ((tile * (tile + 1) / 2 + j) * 2 + e) * 512 + lane * 16;
      };
      if (here) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int j = half + 2 * i;
          if (j > tile) break;
#pragma unroll
          for (int e = 0; e < 2; ++e)
            *reinterpret_cast<float4*>(exchanged(j, e)) = make_float4(G[i][e][0], G[i][e][1], G[i][e][2], G[i][e][3]);
        }
      }
      __syncthreads();
      const int t_low = 16 * tile + g, t_high = t_low + 8;
      const float before_low = before[t_low], before_high = before[t_high];
      double earlier_tiles = 1.;                   // the whole tiles before this one
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j < tile) earlier_tiles *= whole[j];
      const float earlier = (float)earlier_tiles;
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        Y[j][0] *= earlier * before_low;
        Y[j][1] *= earlier * before_low;
        Y[j][2] *= earlier * before_high;
        Y[j][3] *= earlier * before_high;
      }
      // what the chunk's own tokens give: the weights are the first operand as they lie in registers
      double between_tiles = 1.;                   // the whole tiles between s's and t's
#pragma unroll
      for (int kk = 3; kk >= 0; --kk) {
        if (kk > tile || !here) continue;
        uint32_t wf[3][4];
        const float between = (float)between_tiles;
#pragma unroll
        for (int e = 0; e < 2; ++e) {              // the eight tokens s of each half of the 16
          const int s = 8 * e + q2;
          const float4 scores = *reinterpret_cast<const float4*>(exchanged(kk, e));
          const float p[4] = {scores.x, scores.y, scores.z, scores.w};
          float w[4];
          if (kk == tile) {
            const float2 low = *reinterpret_cast<const float2*>(diagonal + t_low * kDiagonalPitch + s);
            const float2 high = *reinterpret_cast<const float2*>(diagonal + t_high * kDiagonalPitch + s);
            w[0] = s <= g ? p[0] * low.x : 0.f;
            w[1] = s + 1 <= g ? p[1] * low.y : 0.f;
            w[2] = s <= g + 8 ? p[2] * high.x : 0.f;
            w[3] = s + 1 <= g + 8 ? p[3] * high.y : 0.f;
          } else {
            const float2 tail = *reinterpret_cast<const float2*>(behind + 16 * kk + s);
            w[0] = p[0] * (before_low * between * tail.x);
            w[1] = p[1] * (before_low * between * tail.y);
            w[2] = p[2] * (before_high * between * tail.x);
            w[3] = p[3] * (before_high * between * tail.y);
          }
          uint32_t part[3];
          split3(w[0], w[1], part);
#pragma unroll
          for (int i = 0; i < 3; ++i) wf[i][2 * e] = part[i];
          split3(w[2], w[3], part);
#pragma unroll
          for (int i = 0; i < 3; ++i) wf[i][2 * e + 1] = part[i];
        }
        if (kk < tile) between_tiles *= whole[kk];
        uint32_t odd = 0;                          // values of this warp's own tokens that are not finite
        auto keep_finite = [&](uint32_t (&v)[kIn][2]) {     // (such a value's other parts are zeros)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t bad = not_finite(v[0][e]);
            odd |= bad;
            v[0][e] &= ~((bad >> 15) * 0xffffu);
          }
        };
#pragma unroll
        for (int j = 0; j < NH / 2; ++j) {
          uint32_t v0[kIn][2], v1[kIn][2];
#pragma unroll
          for (int p = 0; p < kIn; ++p) column_tiles(v0[p], v1[p], L::kValue + p * L::kValuePart, 16 * kk, n0 + 2 * j);
          if (kk == tile) {
            keep_finite(v0);
            keep_finite(v1);
          }
          mma_parts<3, kIn>(Y[2 * j], wf, v0);
          mma_parts<3, kIn>(Y[2 * j + 1], wf, v1);
        }
        if constexpr (NH & 1) {
          uint32_t v0[kIn][2];
#pragma unroll
          for (int p = 0; p < kIn; ++p) column_tile(v0[p], L::kValue + p * L::kValuePart, 16 * kk, n0 + NH - 1);
          if (kk == tile) keep_finite(v0);
          mma_parts<3, kIn>(Y[NH - 1], wf, v0);
        }
        if (kk == tile && __any_sync(0xffffffffu, odd != 0)) {   // what was left out, token after token (seldom: never for finite inputs)
#pragma unroll 1
          for (int quarter = 0; quarter < 4; ++quarter)
#pragma unroll
            for (int place = 0; place < 4; ++place) {
              const int e = place >> 1, s = 8 * e + 2 * quarter + (place & 1);
              auto weight_of = [&](int row_half) {   // of token s for this lane's row, from the lane that made it
                float sum = 0.f;
#pragma unroll
                for (int i = 2; i >= 0; --i)
                  sum += place & 1 ? high_bf16(wf[i][2 * e + row_half]) : low_bf16(wf[i][2 * e + row_half]);
                return __shfl_sync(0xffffffffu, sum, (lane & ~3) | quarter);
              };
              const float w_low = weight_of(0), w_high = weight_of(1);
#pragma unroll
              for (int j = 0; j < NH; ++j) {
                const int row = 16 * tile + s;
                const uint32_t pair = lds_u32(base + L::kValue + row * L::kColPitch + L::column(row, n0 + j) + q2 * 2);
                const uint32_t bad = not_finite(pair);
                if (bad & 0x8000u) {
                  if (s <= g) Y[j][0] = fmaf(w_low, low_bf16(pair), Y[j][0]);
                  if (s <= g + 8) Y[j][2] = fmaf(w_high, low_bf16(pair), Y[j][2]);
                }
                if (bad & 0x80000000u) {
                  if (s <= g) Y[j][1] = fmaf(w_low, high_bf16(pair), Y[j][1]);
                  if (s <= g + 8) Y[j][3] = fmaf(w_high, high_bf16(pair), Y[j][3]);
                }
              }
            }
        }
      }
      float* y_out = a.y + ((long long)t0 * a.heads + head) * vdim;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = e ? t_high : t_low;
        if (t >= n) continue;
#pragma unroll
        for (int j = 0; j < NH; ++j) {
          const int col = column0 + 8 * (n0 + j) + q2;
          if (col >= vdim) continue;
          float2 out = make_float2(Y[j][2 * e], Y[j][2 * e + 1]);
          if (a.skip) {
            const uint32_t at = base + L::kValue + t * L::kColPitch + L::column(t, n0 + j) + q2 * 2;
            float vx = 0.f, vy = 0.f;
#pragma unroll
            for (int p = kIn - 1; p >= 0; --p) {
              const uint32_t raw = lds_u32(at + p * L::kValuePart);
              vx += low_bf16(raw);
              vy += high_bf16(raw);
            }
            out.x = fmaf(skip, vx, out.x);
            out.y = fmaf(skip, vy, out.y);
          }
          *reinterpret_cast<float2*>(y_out + t * y_step + col) = out;
        }
      }
    }

    if (!more && !end_state) break;                // nobody asks for the state behind this chunk
    const double through_chunk = (whole[0] * whole[1]) * (whole[2] * whole[3]);
    const float through = (float)through_chunk;
    decay_product *= through_chunk;
    auto weight = [&](int s) {                     // D[last, s] s_s
      double later = 1.;                           // the whole tiles behind s's
#pragma unroll
      for (int j = 1; j < 4; ++j)
        if (16 * j > s) later *= whole[j];
      return (float)later * behind[s];
    };
    if (kEmit) {
      __syncthreads();                             // everyone has read the state that is replaced here
#pragma unroll
      for (int m = 0; m < kMT; ++m)
#pragma unroll
        for (int j = 0; j < NH; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int row = (tile * kMT + m) * 16 + g + 8 * e;
            const uint32_t at = base + L::kState + row * L::kColPitch + L::column(row, n0 + j) + q2 * 2;
            float x = 0.f, y = 0.f;
#pragma unroll
            for (int p = 2; p >= 0; --p) {         // three parts of 24 bits: the sum is the value they came from
              const uint32_t raw = lds_u32(at + p * L::kStatePart);
              x += low_bf16(raw);
              y += high_bf16(raw);
            }
            S[m][j][2 * e] = x;
            S[m][j][2 * e + 1] = y;
          }
    } else {
      // the weighted values as parts in the values' place, made once for the four warps that use them
      for (int i = threadIdx.x; i < 16 * tiles * (kColumns / 4); i += kChunkThreads) {
        const int s = i / (kColumns / 4), quad = i - s * (kColumns / 4);
        const uint32_t at = base + L::kValue + s * L::kColPitch + L::column(s, quad >> 1) + (quad & 1) * 8;
        float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int p = kIn - 1; p >= 0; --p) {
          const uint2 raw = lds_v2(at + p * L::kValuePart);
          x[0] += low_bf16(raw.x);
          x[1] += high_bf16(raw.x);
          x[2] += low_bf16(raw.y);
          x[3] += high_bf16(raw.y);
        }
        const float w = weight(s);
        uint32_t lo[3], hi[3];
        split3(w * x[0], w * x[1], lo);
        split3(w * x[2], w * x[3], hi);
#pragma unroll
        for (int p = 0; p < 3; ++p) sts_v2(at + p * L::kValuePart, lo[p], hi[p]);
      }
      __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < kMT; ++m)
#pragma unroll
      for (int j = 0; j < NH; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[m][j][e] *= through;
#pragma unroll 1
    for (int kk = 0; kk < tiles; ++kk) {
      uint32_t kf[kMT][kIn][4];
#pragma unroll
      for (int m = 0; m < kMT; ++m)
#pragma unroll
        for (int p = 0; p < kIn; ++p)
          ldsm_x4_trans(kf[m][p], base + L::kKey + p * L::kKeyPart + (16 * kk + in8 + 8 * third) * L::kRowPitch +
                                      ((2 * (tile * kMT + m) + second) ^ in8) * 16);
      float w[4];                                  // of the tokens q2, q2 + 1, q2 + 8, q2 + 9 of the tile
      if (kEmit) {
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = weight(16 * kk + q2 + (e & 1) + 8 * (e >> 1));
      }
      // the weighted values as the second operand: in the emitting pass, which seldom comes here (portions of one
      // segment), made from the values as they are loaded
      auto weighted = [&](uint32_t (&out)[3][2], const uint32_t (&raw)[kUsed][2]) {
        if constexpr (!kEmit) {
#pragma unroll
          for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int e = 0; e < 2; ++e) out[p][e] = raw[p][e];
        } else {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float x = 0.f, y = 0.f;
#pragma unroll
            for (int p = kUsed - 1; p >= 0; --p) {
              x += low_bf16(raw[p][e]);
              y += high_bf16(raw[p][e]);
            }
            uint32_t part[3];
            split3(w[2 * e] * x, w[2 * e + 1] * y, part);
#pragma unroll
            for (int p = 0; p < 3; ++p) out[p][e] = part[p];
          }
        }
      };
#pragma unroll
      for (int j = 0; j < NH / 2; ++j) {
        uint32_t raw0[kUsed][2], raw1[kUsed][2], v0[3][2], v1[3][2];
#pragma unroll
        for (int p = 0; p < kUsed; ++p) column_tiles(raw0[p], raw1[p], L::kValue + p * L::kValuePart, 16 * kk, n0 + 2 * j);
        weighted(v0, raw0);
        weighted(v1, raw1);
#pragma unroll
        for (int m = 0; m < kMT; ++m) {
          mma_parts<kIn, 3>(S[m][2 * j], kf[m], v0);
          mma_parts<kIn, 3>(S[m][2 * j + 1], kf[m], v1);
        }
      }
      if constexpr (NH & 1) {
        uint32_t raw0[kUsed][2], v0[3][2];
#pragma unroll
        for (int p = 0; p < kUsed; ++p) column_tile(raw0[p], L::kValue + p * L::kValuePart, 16 * kk, n0 + NH - 1);
        weighted(v0, raw0);
#pragma unroll
        for (int m = 0; m < kMT; ++m) mma_parts<kIn, 3>(S[m][NH - 1], kf[m], v0);
      }
    }
    if (kEmit && more) {
#pragma unroll
      for (int m = 0; m < kMT; ++m)
#pragma unroll
        for (int j = 0; j < NH; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int row = (tile * kMT + m) * 16 + g + 8 * e;
            const uint32_t at = base + L::kState + row * L::kColPitch + L::column(row, n0 + j) + q2 * 2;
            uint32_t part[3];
            split3(S[m][j][2 * e], S[m][j][2 * e + 1], part);
#pragma unroll
            for (int p = 0; p < 3; ++p) sts_u32(at + p * L::kStatePart, part[p]);
          }
    }
    if (more) __syncthreads();                     // the next chunk's inputs take these ones' place
  }
  if (end_state) {
#pragma unroll
    for (int m = 0; m < kMT; ++m)
#pragma unroll
      for (int j = 0; j < NH; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = (tile * kMT + m) * 16 + g + 8 * e, col = column0 + 8 * (n0 + j) + q2;
          if (row < dim && col < vdim)
            *reinterpret_cast<float2*>(end_state + (long long)row * vdim + col) =
                make_float2(S[m][j][2 * e], S[m][j][2 * e + 1]);
        }
  }
  if (!kEmit && blockIdx.x == 0 && threadIdx.x == 0) a.segment_decay[(long long)blockIdx.z * a.heads + head] = (float)decay_product;
}

// Between the two passes: walk a request's segments, S_start(next) = P S_start + B, leave every segment's start
// state in parts, and write the request's final state into its slot.  Bound by what it reads and writes (4 and 6 bytes an
// element and segment, mostly in the L2).
__global__ void __launch_bounds__(128)
recurrence_chunk_walk_kernel(const __grid_constant__ ChunkArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int head = blockIdx.y;
  int first;
  const int r = find_portion<true>(a, (int)blockIdx.z, &first);
  if (r < 0) return;
  const int count = a.q_start[r + 1] - a.q_start[r];
  const int num_segments = (count + a.segment_len - 1) / a.segment_len;
  if (num_segments <= 1) return;
  const int slot = a.state_slots[r];
  const long long per_head = (long long)a.dim * a.vdim;
  constexpr int kAtOnce = 8;       // segments whose B and P are in registers before the chain of products starts
  for (long long e = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x); e < per_head; e += 4ll * gridDim.x * blockDim.x) {
    float* slot_state = (slot >= 0 && slot < a.num_slots) ? a.state + (long long)slot * a.state_stride + head * per_head + e : nullptr;
    float4 current = slot_state ? *reinterpret_cast<const float4*>(slot_state) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int start = 0; start < num_segments; start += kAtOnce) {
      float4 b[kAtOnce];
      float p[kAtOnce];
  #pragma unroll
      for (int u = 0; u < kAtOnce; ++u) {
        const long long index = ((long long)first + min(start + u, num_segments - 1)) * a.heads + head;
        b[u] = *reinterpret_cast<const float4*>(a.segment_state + index * per_head + e);
        p[u] = a.segment_decay[index];
      }
  #pragma unroll
      for (int u = 0; u < kAtOnce; ++u) {
        if (start + u >= num_segments) break;
        const long long index = ((long long)first + start + u) * a.heads + head;
        uint32_t lo[3], hi[3];
        split3(current.x, current.y, lo);
        split3(current.z, current.w, hi);
  #pragma unroll
        for (int i = 0; i < 3; ++i)
          *reinterpret_cast<uint2*>(a.segment_start + (3 * index + i) * per_head + e) = make_uint2(lo[i], hi[i]);
        current.x = fmaf(p[u], current.x, b[u].x);
        current.y = fmaf(p[u], current.y, b[u].y);
        current.z = fmaf(p[u], current.z, b[u].z);
        current.w = fmaf(p[u], current.w, b[u].w);
      }
    }
    if (slot_state) *reinterpret_cast<float4*>(slot_state) = current;
  }
}

template <int ROWS, int NT, bool kAct, bool kEmit>
static cudaError_t launch_chunks(const ChunkArgs& a, int slots, cudaStream_t stream) {
  constexpr int kBytes = ChunkLayout<ROWS, NT, kAct, kEmit>::kBytes;
  static_assert(kBytes <= 227 * 1024, "a CTA's shared memory");
  auto kernel = recurrence_chunk_kernel<ROWS, NT, kAct, kEmit>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return e;
  const dim3 grid((a.vdim + NT * 8 - 1) / (NT * 8), a.heads, slots);
  return launch_pdl(kernel, grid, dim3(kChunkThreads), kBytes, stream, a);
}

// `slots`: CTAs along z, one per segment number; 0 says that no portion is longer than a segment.
template <int ROWS, int NT, bool kAct>
static cudaError_t run_chunks(const ChunkArgs& a, int portions, int slots, cudaStream_t stream) {
  if (slots == 0) return launch_chunks<ROWS, NT, kAct, true>(a, portions, stream);
  cudaError_t e = launch_chunks<ROWS, NT, kAct, false>(a, slots, stream);
  if (e != cudaSuccess) return e;
  // portions of one segment have nothing to walk: with many portions the CTAs of one take more each
  const long long blocks = ((long long)a.dim * a.vdim / 4 + 127) / 128, most = 1 + 4096 / ((long long)a.heads * portions);
  e = launch_pdl(recurrence_chunk_walk_kernel, dim3((unsigned)(blocks < most ? blocks : most), a.heads, portions), dim3(128),
                 0, stream, a);
  if (e != cudaSuccess) return e;
  return launch_chunks<ROWS, NT, kAct, true>(a, slots, stream);
}

}  // namespace einf

using namespace einf;

// q, k, v: bfloat16, 8-byte aligned rows (strides and sizes in multiples of four elements), the state 16-byte aligned; dim
// up to 128.  Portions of min_len tokens and more are taken, `portions` of them at most.  `slots`: 0 where none of them is
// longer than segment_len; else tokens / segment_len + portions, with segment_len a multiple of 64.  `tiles`: columns of the
// state that a CTA takes, in eights (4 or 8; 10 where dim is 64 at most).
extern "C" int einf_linear_recurrence_chunks(const void* q, const void* k, const void* v, long long q_stride,
                                             long long k_stride, long long v_stride, const float* head_decay,
                                             const float* token_decay, const float* token_scale, const float* skip,
                                             float* state, long long state_stride, int num_slots, const int* q_start,
                                             const int* state_slots, int num_requests, int portions, int min_len, float* y,
                                             int heads, int groups, int dim, int vdim, int act, int tiles, int slots,
                                             int segment_len,
                                             float* segment_state, void* segment_start, float* segment_decay,
                                             cudaStream_t stream) {
  if (num_requests == 0 || portions == 0) return 0;
  if (heads <= 0 || groups <= 0 || heads % groups || dim <= 0 || dim > 128 || dim % 4 || vdim <= 0 || vdim % 4 ||
      heads > 65535 || portions < 0 || portions > 65535 || min_len < 1 || slots < 0 || slots > 65535 || segment_len < 1 ||
      (slots && (!segment_state || !segment_start || !segment_decay || segment_len % kChunk)) || state_stride % 4 ||
      ((uintptr_t)state & 15) || ((uintptr_t)y & 7) || ((uintptr_t)q & 7) || ((uintptr_t)k & 7) || ((uintptr_t)v & 7) ||
      q_stride % 4 || k_stride % 4 || v_stride % 4)
    return (int)cudaErrorInvalidValue;
  ChunkArgs a = {};
  a.q = (const __nv_bfloat16*)q; a.k = (const __nv_bfloat16*)k; a.v = (const __nv_bfloat16*)v;
  a.q_stride = q_stride; a.k_stride = k_stride; a.v_stride = v_stride;
  a.head_decay = head_decay; a.token_decay = token_decay; a.token_scale = token_scale; a.skip = skip;
  a.state = state; a.state_stride = state_stride;
  a.q_start = q_start; a.state_slots = state_slots;
  a.y = y;
  a.segment_state = segment_state; a.segment_start = (__nv_bfloat16*)segment_start; a.segment_decay = segment_decay;
  a.num_slots = num_slots; a.heads = heads; a.groups = groups; a.dim = dim; a.vdim = vdim;
  a.num_requests = num_requests; a.min_len = min_len;
  a.segment_len = slots ? segment_len : 1 << 30;     // one segment each: numbered by the portions alone
  a.wide = (!((uintptr_t)q & 15) && q_stride % 8 == 0 && dim % 8 == 0 ? 1 : 0) |
           (!((uintptr_t)k & 15) && k_stride % 8 == 0 && dim % 8 == 0 ? 2 : 0) |
           (!((uintptr_t)v & 15) && v_stride % 8 == 0 && vdim % 8 == 0 ? 4 : 0) | (vdim % 8 == 0 ? 8 : 0);
#define EINF_CHUNKS(ROWS_, NT_)                                                                                  \
  if (dim <= ROWS_ && tiles == NT_)                                                                             \
    return act ? (int)run_chunks<ROWS_, NT_, true>(a, portions, slots, stream)                                  \
               : (int)run_chunks<ROWS_, NT_, false>(a, portions, slots, stream);
  EINF_CHUNKS(64, 4)
  EINF_CHUNKS(64, 8)
  EINF_CHUNKS(64, 10)
  EINF_CHUNKS(128, 4)
  EINF_CHUNKS(128, 8)
#undef EINF_CHUNKS
  return (int)cudaErrorInvalidValue;
}
