// out[T, N] = X[T, K] . W[N, K]^T (+ bias) in bfloat16 on the fifth-generation tensor
// cores: TMA loads, tcgen05.mma with the accumulator in tensor memory, split-K.
//
// The weight matrix is the 128-row operand of the MMA and the tokens are its N
// dimension (16 to 256 wide), so a decode step with a handful of tokens still
// issues full-rate instructions and the kernel is what it should be there: a
// stream of W through shared memory at HBM speed.  One CTA owns one
// (128 weight rows) x (token tile) x (K range) block:
//
//   warp 0   producer: one lane issues the TMA loads of the W and X tiles of each
//            64-wide K block into a ring of shared-memory stages (128-byte swizzle);
//            the W tiles of the first stages are requested before the wait on the
//            previous kernel (weights do not depend on it), the X tiles after it
//   warp 1   allocates tensor memory; one lane issues four tcgen05.mma (K = 16 each)
//            per stage and commits the stage back to the producer
//   warps 2-5 epilogue: tcgen05.ld the accumulator (lane = weight row, column =
//            token), add the bias, store transposed into out[token, row]
//
// With split-K the CTAs of one output block each take a K range and write 32-bit
// partial sums [split, T, N]; the consumer (the norm, rotary or activation kernel
// that follows) adds them up, so no atomics and no extra pass are needed and the
// result does not depend on timing.  Every wait on a barrier is bounded; a wait
// that gives up sets a bit in the status word and the CTA drains and leaves.
//
// No multicast anywhere: every CTA fetches its own tiles.
// (replaces the library products of the reference: F.linear at
// src/einf/executors/torch/packed_qkv.py:148 and qwen.py:207-208,489,773.)
#include <cuda.h>

#include "common.cuh"

namespace einf {

constexpr int kBlockW = 128;    // weight rows per CTA (UMMA M)
constexpr int kBlockK = 64;     // K per stage: 64 bf16 = 128 bytes = one swizzle span
constexpr int kUmmaK = 16;
constexpr int kGemmThreads = 192;
constexpr int kMaxStages = 8;
constexpr int kWTileBytes = kBlockW * kBlockK * 2;   // 16 KB
constexpr int kMaxPolls = 1 << 22;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded wait: false (and a status bit) if the phase did not complete in time.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status) {
  for (int poll = 0; poll < kMaxPolls; ++poll) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  atomicOr(status, kStatusWaitExpired);
  return false;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: rows of 128
// bytes, eight rows per 1024-byte group (stride byte offset 1024), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
  uint64_t desc = (addr >> 4) & 0x3FFFu;
  desc |= (uint64_t)1 << 16;              // leading byte offset: unused for swizzled K-major, 1 by convention
  desc |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset
  desc |= (uint64_t)1 << 46;              // version
  desc |= (uint64_t)2 << 61;              // 128-byte swizzle
  return desc;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

struct GemmParams {
  void* out;            // [T, N] (out_dtype), or 32-bit partial sums [splits, T, N] when splits > 1
  const float* bias;    // [N] or null (with split-K it is added by split 0)
  int* status;
  int tokens, n, k;
  int token_tile;       // BN: 16 .. 256, a multiple of 16
  int stages;
  int kblocks_per_split;
  int out_dtype;        // kFloat32 | kBFloat16 (ignored with split-K)
  long long ldo;        // row stride of out in elements
};

__global__ void __launch_bounds__(kGemmThreads)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                    GemmParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // Stage ring first (1024-byte aligned tiles), barriers after it.
  const uint32_t smem_base = (smem_addr(smem_raw) + 1023u) & ~1023u;
  const int x_tile_bytes = p.token_tile * kBlockK * 2;
  const int stage_bytes = kWTileBytes + x_tile_bytes;
  const uint32_t bar_base = smem_base + p.stages * stage_bytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
  const uint32_t accum_bar = bar_base + 8u * (2 * kMaxStages);
  const uint32_t tmem_holder = bar_base + 8u * (2 * kMaxStages + 1);
  unsigned char* generic_base = smem_raw + (smem_base - smem_addr(smem_raw));
  volatile uint32_t* tmem_holder_ptr =
      reinterpret_cast<volatile uint32_t*>(generic_base + p.stages * stage_bytes + 8 * (2 * kMaxStages + 1));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kBlockW;
  const int t0 = blockIdx.y * p.token_tile;
  const int split = blockIdx.z, splits = gridDim.z;
  const int total_kblocks = (p.k + kBlockK - 1) / kBlockK;
  const int kb_begin = split * p.kblocks_per_split;
  const int kb_end = min(total_kblocks, kb_begin + p.kblocks_per_split);
  const int num_kblocks = kb_end - kb_begin;   // >= 1 by construction of the grid

  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)p.token_tile) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(accum_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_holder), "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder_ptr;
  // The next kernel may start its own prologue now (it waits for this grid's completion before it
  // touches anything this grid writes).  Not earlier: a kernel that is resident holds its tensor
  // memory, and this one must have its own before a later one can take columns on this SM.
  pdl_launch_dependents();

  if (warp == 0) {
    if (lane == 0) {
      // ---- producer ----
      const int first = min(p.stages, num_kblocks);
      for (int i = 0; i < first; ++i) {   // weights do not depend on the kernel before this one
        mbar_expect_tx(full_bar(i), stage_bytes);
        tma_load_2d(smem_base + i * stage_bytes, &map_w, (kb_begin + i) * kBlockK, n0, full_bar(i));
      }
      pdl_wait();
      for (int i = 0; i < first; ++i)
        tma_load_2d(smem_base + i * stage_bytes + kWTileBytes, &map_x, (kb_begin + i) * kBlockK, t0, full_bar(i));
      bool ok = true;
      for (int i = first; i < num_kblocks && ok; ++i) {
        const int s = i % p.stages;
        ok = mbar_wait(empty_bar(s), ((i / p.stages) & 1) ^ 1, p.status);
        if (!ok) break;
        mbar_expect_tx(full_bar(s), stage_bytes);
        tma_load_2d(smem_base + s * stage_bytes, &map_w, (kb_begin + i) * kBlockK, n0, full_bar(s));
        tma_load_2d(smem_base + s * stage_bytes + kWTileBytes, &map_x, (kb_begin + i) * kBlockK, t0, full_bar(s));
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issuer ----
      // Instruction descriptor: D = F32, A = B = BF16, both K-major, N = token tile, M = 128.
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.token_tile >> 3) << 17) |
                             ((uint32_t)(kBlockW >> 4) << 24);
      bool ok = true;
      pdl_wait();   // bounded waits start once only this kernel's own progress is waited for
      for (int i = 0; i < num_kblocks && ok; ++i) {
        const int s = i % p.stages;
        ok = mbar_wait(full_bar(s), (i / p.stages) & 1, p.status);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // descriptors once per stage, then one add on the low word per MMA (the address field is
        // in units of 16 bytes and cannot overflow: shared memory ends below 256 KB)
        const uint64_t w_desc = umma_desc(smem_base + s * stage_bytes);
        const uint64_t x_desc = umma_desc(smem_base + s * stage_bytes + kWTileBytes);
#pragma unroll
        for (int kk = 0; kk < kBlockK / kUmmaK; ++kk) {
          const uint32_t step = (uint32_t)(kk * kUmmaK * 2) >> 4;
          umma_bf16(tmem_base, (w_desc & 0xFFFFFFFF00000000ull) | (uint32_t)((uint32_t)w_desc + step),
                    (x_desc & 0xFFFFFFFF00000000ull) | (uint32_t)((uint32_t)x_desc + step), idesc,
                    (i > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(empty_bar(s));   // the stage is free once these MMAs have read it
      }
      umma_commit(accum_bar);        // the accumulator is complete once every MMA is
    }
  } else {
    // ---- epilogue: warps 2..5 own tensor-memory lanes 32 * (warp % 4) .. + 31 ----
    pdl_wait();   // as above
    const bool ok = mbar_wait(accum_bar, 0, p.status);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
      const int lane_base = (warp & 3) * 32;
      const int row = n0 + lane_base + lane;         // weight row = output column
      const bool row_ok = row < p.n;
      const bool partial = splits > 1;
      const float bias = (p.bias && row_ok && split == 0) ? p.bias[row] : 0.f;
      float* out_f = partial ? reinterpret_cast<float*>(p.out) + (size_t)split * p.tokens * p.ldo
                             : reinterpret_cast<float*>(p.out);
      __nv_bfloat16* out_h = reinterpret_cast<__nv_bfloat16*>(p.out);
      const bool as_float = partial || p.out_dtype == kFloat32;
      // One store per (token, weight row), 128 bytes per warp.  Kept to a pointer bump and a store
      // per column: with an index computation and a bounds test per element this loop, which
      // one warp per 32 rows runs alone, took longer than the product itself at 64 tokens.
      for (int col0 = 0; col0 < p.token_tile; col0 += 16) {
        const int t_first = t0 + col0;
        if (t_first >= p.tokens) break;              // uniform across the warp
        uint32_t v[16];
        tmem_load16(tmem_base + ((uint32_t)lane_base << 16) + (uint32_t)col0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row_ok) {
          const int valid = min(16, p.tokens - t_first);
          if (as_float) {
            float* dst = out_f + (size_t)t_first * p.ldo + row;
            if (valid == 16) {
#pragma unroll
              for (int c = 0; c < 16; ++c, dst += p.ldo) *dst = __uint_as_float(v[c]) + bias;
            } else {
#pragma unroll
              for (int c = 0; c < 16; ++c, dst += p.ldo)
                if (c < valid) *dst = __uint_as_float(v[c]) + bias;
            }
          } else {
            __nv_bfloat16* dst = out_h + (size_t)t_first * p.ldo + row;
#pragma unroll
            for (int c = 0; c < 16; ++c, dst += p.ldo)
              if (c < valid) *dst = __float2bfloat16_rn(__uint_as_float(v[c]) + bias);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

// ---------------------------------------------------------------------------
// The same product over rows that are sorted by group (the experts of a routed feed-forward):
// out[r] = W[g] x[r] for offsets[g] <= r < offsets[g + 1], W stacked [groups, n, k].  The grid's y
// dimension is a list of token tiles that never cross a group: tile slot y belongs to the group
// and the place that a walk over the offsets gives it (slots beyond the last tile leave at once),
// so the host never has to know how many rows a group got.  A tile's boxes of x may reach into the
// next group's rows (or past the end, where TMA fills zeros): columns of the accumulator from the tile's rows on are at most
// 15, and not stored.  With `splits` > 1 (grid z) the CTAs of a tile each take a K range and write
// 32-bit partial sums [splits, rows, n] that the consumer adds up in order (a matrix with few row
// tiles and a handful of rows per group would otherwise run on a third of the GPU).
// ---------------------------------------------------------------------------
struct GroupedParams {
  void* out;              // [rows, n] (out_dtype), or float partial sums [splits, rows, n]
  int kblocks_per_split;
  const int* offsets;     // [groups + 1], written by a kernel earlier in the step
  int* status;
  int rows, n, k, groups;
  int token_tile;
  int box;                // rows of x a load brings
  int stages;
  int out_dtype;
};

// A group's tiles are of one size, as near as multiples of 16 allow: 520 rows are three tiles of 176, not two of 256 and one
// of 8, which would read the whole weight tile for its 8 rows.
__device__ __forceinline__ bool find_group_tile(const GroupedParams& p, int slot, int* group, int* t0, int* valid) {
  for (int g = 0; g < p.groups; ++g) {
    const int begin = p.offsets[g], count = p.offsets[g + 1] - begin;
    const int tiles = (count + p.token_tile - 1) / p.token_tile;
    if (slot < tiles) {
      const int each = min(p.token_tile, ((count + tiles - 1) / tiles + 15) / 16 * 16);
      *group = g;
      *t0 = begin + slot * each;
      *valid = min(each, count - slot * each);
      return *valid > 0;
    }
    slot -= tiles;
  }
  return false;
}

__global__ void __launch_bounds__(kGemmThreads)
gemm_grouped_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                            GroupedParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t smem_base = (smem_addr(smem_raw) + 1023u) & ~1023u;
  const int x_tile_bytes = p.token_tile * kBlockK * 2;
  const int stage_bytes = kWTileBytes + x_tile_bytes;
  const uint32_t bar_base = smem_base + p.stages * stage_bytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
  const uint32_t accum_bar = bar_base + 8u * (2 * kMaxStages);
  const uint32_t tmem_holder = bar_base + 8u * (2 * kMaxStages + 1);
  unsigned char* generic_base = smem_raw + (smem_base - smem_addr(smem_raw));
  volatile uint32_t* tmem_holder_ptr =
      reinterpret_cast<volatile uint32_t*>(generic_base + p.stages * stage_bytes + 8 * (2 * kMaxStages + 1));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kBlockW;
  const int split = blockIdx.z, splits = gridDim.z;
  const int total_kblocks = (p.k + kBlockK - 1) / kBlockK;
  const int kb_begin = split * p.kblocks_per_split;
  const int num_kblocks = min(total_kblocks, kb_begin + p.kblocks_per_split) - kb_begin;   // >= 1 by the grid
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)p.token_tile) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(accum_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_holder), "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder_ptr;
  pdl_launch_dependents();

  // Every role finds the tile by itself, after the wait for the kernel that wrote the offsets.
  pdl_wait();
  int group = 0, t0 = 0, valid = 0;
  const bool have = find_group_tile(p, blockIdx.y, &group, &t0, &valid);

  const int boxes = (valid + p.box - 1) / p.box;       // of x: the rows of this tile alone
  const int load_bytes = kWTileBytes + boxes * p.box * kBlockK * 2;

  if (have && warp == 0) {
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < num_kblocks && ok; ++i) {
        const int s = i % p.stages;
        if (i >= p.stages) ok = mbar_wait(empty_bar(s), ((i / p.stages) & 1) ^ 1, p.status);
        if (!ok) break;
        mbar_expect_tx(full_bar(s), load_bytes);
        tma_load_2d(smem_base + s * stage_bytes, &map_w, (kb_begin + i) * kBlockK, group * p.n + n0, full_bar(s));
        for (int b = 0; b < boxes; ++b)
          tma_load_2d(smem_base + s * stage_bytes + kWTileBytes + b * p.box * kBlockK * 2, &map_x, (kb_begin + i) * kBlockK,
                      t0 + b * p.box, full_bar(s));
      }
    }
  } else if (have && warp == 1) {
    if (lane == 0) {
      const int columns = (valid + 15) / 16 * 16;      // the products' N: this tile's rows
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(columns >> 3) << 17) |
                             ((uint32_t)(kBlockW >> 4) << 24);
      bool ok = true;
      for (int i = 0; i < num_kblocks && ok; ++i) {
        const int s = i % p.stages;
        ok = mbar_wait(full_bar(s), (i / p.stages) & 1, p.status);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t w_desc = umma_desc(smem_base + s * stage_bytes);
        const uint64_t x_desc = umma_desc(smem_base + s * stage_bytes + kWTileBytes);
#pragma unroll
        for (int kk = 0; kk < kBlockK / kUmmaK; ++kk) {
          const uint32_t step = (uint32_t)(kk * kUmmaK * 2) >> 4;
          umma_bf16(tmem_base, (w_desc & 0xFFFFFFFF00000000ull) | (uint32_t)((uint32_t)w_desc + step),
                    (x_desc & 0xFFFFFFFF00000000ull) | (uint32_t)((uint32_t)x_desc + step), idesc,
                    (i > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(empty_bar(s));
      }
      umma_commit(accum_bar);
    }
  } else if (have) {
    const bool ok = mbar_wait(accum_bar, 0, p.status);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
      const int lane_base = (warp & 3) * 32;
      const int row = n0 + lane_base + lane;         // weight row of this group = output column
      const bool row_ok = row < p.n;
      float* out_f = reinterpret_cast<float*>(p.out) + (splits > 1 ? (size_t)split * p.rows * p.n : 0);
      __nv_bfloat16* out_h = reinterpret_cast<__nv_bfloat16*>(p.out);
      const bool as_float = splits > 1 || p.out_dtype == kFloat32;
      for (int col0 = 0; col0 < p.token_tile; col0 += 16) {
        if (col0 >= valid) break;                    // uniform across the warp
        uint32_t v[16];
        tmem_load16(tmem_base + ((uint32_t)lane_base << 16) + (uint32_t)col0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row_ok) {
          const int count = min(16, valid - col0);
          const size_t first = (size_t)(t0 + col0) * p.n + row;
          if (as_float) {
            float* dst = out_f + first;
#pragma unroll
            for (int c = 0; c < 16; ++c, dst += p.n)
              if (c < count) *dst = __uint_as_float(v[c]);
          } else {
            __nv_bfloat16* dst = out_h + first;
#pragma unroll
            for (int c = 0; c < 16; ++c, dst += p.n)
              if (c < count) *dst = __float2bfloat16_rn(__uint_as_float(v[c]));
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

}  // namespace einf

using namespace einf;

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &result) != cudaSuccess ||
        result != cudaDriverEntryPointSuccess)
      return (EncodeTiledFn) nullptr;
    return (EncodeTiledFn)ptr;
  }();
  return fn;
}

// A [rows, k] bfloat16 matrix with unit stride along k, as a TMA map with a (64 x box_rows) box.
static int make_map(CUtensorMap* map, const void* base, long long rows, long long k, long long row_stride_elems,
                    int box_rows) {
  EncodeTiledFn encode = encode_tiled();
  if (!encode) return (int)cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)row_stride_elems * 2};
  cuuint32_t box[2] = {(cuuint32_t)kBlockK, (cuuint32_t)box_rows};
  cuuint32_t element_strides[2] = {1, 1};
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
                      element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

// Shared memory the kernel needs for a token tile and a number of stages.
static size_t smem_bytes(int token_tile, int stages) {
  return 1024 + (size_t)stages * (kWTileBytes + token_tile * kBlockK * 2) + 8 * (2 * kMaxStages + 2);
}

// The token tile the launcher picks for `tokens` rows: the smallest multiple of 16 that holds
// them, 256 at most.
extern "C" int einf_gemm_tcgen05_token_tile(int tokens) {
  int tile = (tokens + 15) / 16 * 16;
  return tile < 16 ? 16 : (tile > 256 ? 256 : tile);
}

// x: [tokens, k] bfloat16, row stride ldx; w: [n, k] bfloat16 contiguous; out as GemmParams says.
// k must be a multiple of 8 and both base pointers 16-byte aligned (TMA rules).
// splits > 1: out holds 32-bit partial sums [splits, tokens, n] (ldo = n).
extern "C" int einf_gemm_tcgen05(const void* x, const void* w, const float* bias, void* out, int out_dtype,
                                 int tokens, int n, int k, long long ldx, long long ldo, int splits, int* status,
                                 cudaStream_t stream) {
  if (tokens == 0 || n == 0) return 0;
  if (k % 8 != 0 || ldx % 8 != 0 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return (int)cudaErrorInvalidValue;
  const int total_kblocks = (k + kBlockK - 1) / kBlockK;
  if (splits < 1) splits = 1;
  if (splits > total_kblocks) splits = total_kblocks;
  int per_split = (total_kblocks + splits - 1) / splits;
  splits = (total_kblocks + per_split - 1) / per_split;   // no empty split
  const int token_tile = einf_gemm_tcgen05_token_tile(tokens);
  // Two CTAs per SM when the stages allow it (about 110 KB each): one streams while the
  // other runs its epilogue.  Never fewer than three stages for a long K range.
  int stages = per_split < kMaxStages ? per_split : kMaxStages;
  while (stages > 3 && smem_bytes(token_tile, stages) > 110 * 1024) --stages;
  while (stages > 1 && smem_bytes(token_tile, stages) > 200 * 1024) --stages;
  CUtensorMap map_w, map_x;
  int rc = make_map(&map_w, w, n, k, k, kBlockW);
  if (rc) return rc;
  rc = make_map(&map_x, x, tokens, k, ldx, token_tile);
  if (rc) return rc;
  GemmParams p;
  p.out = out;
  p.bias = bias;
  p.status = status;
  p.tokens = tokens;
  p.n = n;
  p.k = k;
  p.token_tile = token_tile;
  p.stages = stages;
  p.kblocks_per_split = per_split;
  p.out_dtype = out_dtype;
  p.ldo = ldo;
  const size_t smem = smem_bytes(token_tile, stages);
  cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  dim3 grid((n + kBlockW - 1) / kBlockW, (tokens + token_tile - 1) / token_tile, splits);
  return (int)launch_pdl(gemm_tcgen05_kernel, grid, dim3(kGemmThreads), smem, stream, map_w, map_x, p);
}

// Number of splits the launcher will really use for a request of `splits`.
extern "C" int einf_gemm_tcgen05_splits(int k, int splits) {
  const int total_kblocks = (k + kBlockK - 1) / kBlockK;
  if (splits < 1) splits = 1;
  if (splits > total_kblocks) splits = total_kblocks;
  const int per_split = (total_kblocks + splits - 1) / splits;
  return (total_kblocks + per_split - 1) / per_split;
}

// The largest token tile of the grouped product for `rows` rows over `groups` groups of n outputs: about one and a half
// times the average rows of a group, a multiple of 16 between 16 and 128, above that 192 or 256.  The CTAs' reads of W and x
// out of L2 bound the product at many rows (2.6 GB at tiles of 128 for the sizes below, 2 GB at 256), so a weight tile meets
// as many rows as its accumulator holds with two CTAs an SM, one's epilogue beside the other's products.
// Measured (B200): both products of 4,096 rows on eight experts, n and k of 17,920 and 1,536 and of 1,536 and 8,960:
// 218 -> 182 us.  Not where tiles of 128 are one wave of CTAs or less (two an SM): fewer and larger tiles then leave
// multiprocessors empty, and the ring of a larger tile has two stages where that of 128 rows has three.  Eight experts, n
// 1,536, k 8,960, us with 128 / larger: 100 rows an expert (96 CTAs of 128) 80 / 100, 200 (192) 82 / 119, 340 (288) 84 / 113, 512
// (384) 139 / 123; sixteen, n 1,024, k 896: 160 (256) 20.5 / 22.5, 340 (384) 33 / 25; sixty, n 2,816, k 2,048: 160 (2,640) 217 / 193.
extern "C" int einf_gemm_grouped_tcgen05_token_tile(int rows, int groups, int n) {
  const int average = (rows + groups - 1) / (groups > 0 ? groups : 1);
  const int tile = (average * 3 / 2 + 15) / 16 * 16;
  if (tile <= 128) return tile < 16 ? 16 : tile;
  const long long ctas = (long long)((n + kBlockW - 1) / kBlockW) * groups * ((average + 127) / 128);
  if (ctas <= 2 * 148) return 128;
  return tile <= 192 ? 192 : 256;
}

// x: [rows, k] bfloat16 contiguous, sorted by group; w: [groups, n, k] bfloat16 contiguous; offsets: [groups + 1]
// on the device; out: [rows, n] in out_dtype.  k must be a multiple of 8, the base pointers 16-byte aligned.
extern "C" int einf_gemm_grouped_tcgen05(const void* x, const void* w, const int* offsets, void* out, int out_dtype,
                                         int rows, int groups, int n, int k, int splits, int* status,
                                         cudaStream_t stream) {
  if (rows == 0 || n == 0 || groups == 0) return 0;
  if (k % 8 != 0 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return (int)cudaErrorInvalidValue;
  const int token_tile = einf_gemm_grouped_tcgen05_token_tile(rows, groups, n);
  const int total_kblocks = (k + kBlockK - 1) / kBlockK;
  if (splits != einf_gemm_tcgen05_splits(k, splits)) return (int)cudaErrorInvalidValue;   // the caller sized out for it
  const int per_split = (total_kblocks + splits - 1) / splits;
  int stages = per_split < kMaxStages ? per_split : kMaxStages;
  while (stages > 2 && smem_bytes(token_tile, stages) > 110 * 1024) --stages;      // two CTAs an SM
  CUtensorMap map_w, map_x;
  int rc = make_map(&map_w, w, (long long)groups * n, k, k, kBlockW);
  if (rc) return rc;
  const int box = token_tile <= 128 ? token_tile : 64;
  rc = make_map(&map_x, x, rows, k, k, box);
  if (rc) return rc;
  GroupedParams p;
  p.out = out;
  p.offsets = offsets;
  p.status = status;
  p.rows = rows;
  p.n = n;
  p.k = k;
  p.groups = groups;
  p.token_tile = token_tile;
  p.box = box;
  p.stages = stages;
  p.out_dtype = out_dtype;
  p.kblocks_per_split = per_split;
  const size_t smem = smem_bytes(token_tile, stages);
  cudaError_t e = cudaFuncSetAttribute(gemm_grouped_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int slots = (rows + token_tile - 1) / token_tile + (groups < rows ? groups : rows);
  dim3 grid((n + kBlockW - 1) / kBlockW, slots, splits);
  return (int)launch_pdl(gemm_grouped_tcgen05_kernel, grid, dim3(kGemmThreads), smem, stream, map_w, map_x, p);
}
