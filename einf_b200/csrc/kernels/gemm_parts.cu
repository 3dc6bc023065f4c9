// out[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) for 32-bit operands and a 32-bit result on the fifth-generation tensor cores
// (gemm_simt.cu has the FMA product for operands of mixed type and rows that are not aligned).
//
// A 32-bit value is the sum of three bfloat16 parts (8 bits of the significand each), so a product of two is nine bfloat16
// products, of which the six largest count: what is left out is 2^-24 of a term at most.  The instruction cuts its sums
// off where FMA rounds them, so a chain of it drifts.  Therefore 32 elements of K are summed at a time, products of the
// smaller parts first, into a tensor-memory accumulator that starts at zero, and its result is added to a running sum in
// registers by a rounded addition; every 512 elements that sum joins a total in tensor memory.  Error against 64 bits (2-norm, 1 to 2,048
// rows against 896, this / FMA, in 1e-7): normal values, K = 896 0.83 to 0.97 / 2.8, 4,864 0.95 to 1.14 / 3.0, 18,944 1.2 / 3.3;
// where all terms are positive (normal values' magnitudes, uniform ones) 0.64 to 0.76 / 1.1 to 1.3, 0.66 to 0.78 / 0.87, 0.66 to 0.72 / 1.34, or
// 1.08 by one CTA each (64 elements at a time 1.8; without the total 2.1 at 4,864).
//
// A CTA has 128 rows of W (the instruction's M) and 128 rows of A (its N).  Its sixteen warps read the next 64 columns of
// both operands into registers, split them and write the parts into swizzled K-major tiles (two stages of 96 KB), one
// thread issues the 24 products, and while they run the warps split the 64 columns after.  Bound by shared memory: the 24
// products read 192 KB of it and the parts are 96 KB to write, 2,300 cycles at 128 bytes each; 64 columns take 3,200.  (Eight warps
// of twice the work each 90 us where this takes 84.)  Where the tiles are too few for the GPU, CTAs share K and a second
// kernel adds their sums in order.
//
// Measured (B200, us, FMA before): 545 rows, 896 -> 1,152 42 -> 21, 896 -> 896 41 -> 18, 896 -> 9,728 211 -> 84 (113 TFLOP/s),
// 4,864 -> 896 118 -> 45; 2,048 rows, 3,584 -> 4,608 1,300 -> 395 (171 TFLOP/s); one row, 896 -> 9,728 40 -> 26.
//
// A value that is not finite, rounds to infinity as bfloat16 or has bits below the smallest bfloat16 (values below 2^-110) has no
// such parts.  The outputs of its row, and any whose sum is not finite (products of parts may overflow where the operands'
// does not, or to the other infinity), are computed by FMA, the CTA's tile out of shared memory with sums over 256 elements;
// the outputs beside them keep theirs.  (NaN needs no second sum: its first part is NaN.)  545 rows, 896 -> 9,728, one of them with
// an infinity: 172 us (FMA alone 210; 8,050 where every thread walked its outputs by itself), all of them 719, with NaN 88.
#include "mma_sync.cuh"
#include "tcgen05.cuh"

namespace einf {

constexpr int kPartRows = 128, kPartK = 64, kPartThreads = 512;
constexpr int kPartTile = kPartRows * kPartK * 2;                 // bytes of one part of one operand
constexpr int kPartStage = 6 * kPartTile;                         // W's parts, then A's
constexpr int kPartSmem = 2 * kPartStage + 1024;
constexpr int kPartFold = 8;                                      // blocks of 64 columns whose sums are added up before they join the total

struct PartsArgs {
  const float* a; const float* w; const float* bias;
  float* out;                 // [m, n], rows ldo apart; or sums [shares][m][n]
  int m, n, k;
  long long lda, ldo;
  int blocks_each;            // blocks of 64 columns that a CTA takes
  int shared;
  int* status;                // may be null
};

// Eight values as four pairs of each part; false if one is not the sum of its parts (an infinity or a NaN on the way is not).
__device__ __forceinline__ bool split_eight(const float4& x, const float4& y, uint4 (&part)[3]) {
  const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  uint32_t left = 0;                   // of the third parts: bits that bfloat16 has not (NaN, as it is made, has them all)
  uint32_t p[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = v[2 * i], b = v[2 * i + 1];
    p[0][i] = pack_pair(a, b);
    a -= low_bf16(p[0][i]);
    b -= high_bf16(p[0][i]);
    p[1][i] = pack_pair(a, b);
    a -= low_bf16(p[1][i]);
    b -= high_bf16(p[1][i]);
    p[2][i] = pack_pair(a, b);
    left |= __float_as_uint(a) | __float_as_uint(b);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) part[j] = make_uint4(p[j][0], p[j][1], p[j][2], p[j][3]);
  return (left & 0xffffu) == 0u;
}

__device__ __forceinline__ float* parts_out(const PartsArgs& g, int row, int col) {
  return g.out + (g.shared ? (long long)blockIdx.z * g.m * g.n + (long long)row * g.n : (long long)row * g.ldo) + col;
}

// Enters a thread's marked rows among the tile's; those with a NaN, which the thread's columns are looked through for, apart.
__device__ __noinline__ void parts_mark(const PartsArgs& g, uint32_t marks, int row0, int col0, int first, int k1, uint32_t* odd, uint32_t* nan) {
  for (int j = 0; j < 4; ++j) {
    if (!(marks >> j & 1u)) continue;
    const int row = (j & 1 ? row0 : col0) + 64 * (j >> 1);
    const float* from = j & 1 ? g.a + (long long)row * g.lda : g.w + (long long)row * g.k;
    bool is_nan = false;
    for (int at = first; at < k1; at += kPartK)
      for (int e = 0; e < 8; ++e) is_nan = is_nan || from[at + e] != from[at + e];
    atomicOr((is_nan ? nan : odd) + (j & 1) * 4 + (row % kPartRows >> 5), 1u << (row & 31));
  }
}

// Outputs of the CTA's tile over the columns from `first` to k1 by FMA: of this thread's 32 (one row of W, 32 rows of A) those marked
// in `again`.  32 columns of both operands at a time in shared memory, rows side by side.
__device__ __noinline__ void parts_by_fma(const PartsArgs& g, float* w_tile, int row0, int col0, int first, int k1, uint32_t again) {
  constexpr int kStep = 32, kPitch = kPartRows + 4;
  float* a_tile = w_tile + kStep * kPitch;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = tid >> 2, part = (tid & 3) * 8;
  const int col = col0 + (warp & 3) * 32 + lane, first_token = row0 + (warp >> 2) * 32;
  const bool busy = __any_sync(0xffffffffu, again != 0u);     // a warp with nothing to do only brings its share
  const bool w_real = col0 + row < g.n, a_real = row0 + row < g.m;
  const float* w_row = g.w + (long long)(col0 + row) * g.k;
  const float* a_row = g.a + (long long)(row0 + row) * g.lda;
  float block[32], folded[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) block[e] = folded[e] = 0.f;
#pragma unroll 1
  for (int k0 = first; k0 < k1; k0 += kStep) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int at = k0 + part + e;
      w_tile[(part + e) * kPitch + row] = w_real && at < k1 ? w_row[at] : 0.f;
      a_tile[(part + e) * kPitch + row] = a_real && at < k1 ? a_row[at] : 0.f;
    }
    __syncthreads();
#pragma unroll 2
    for (int kk = 0; kk < (busy ? kStep : 0); ++kk) {
      const float w = w_tile[kk * kPitch + (warp & 3) * 32 + lane];
      const float4* a = reinterpret_cast<const float4*>(a_tile + kk * kPitch + (warp >> 2) * 32);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 x = a[e];
        block[4 * e] = fmaf(x.x, w, block[4 * e]);
        block[4 * e + 1] = fmaf(x.y, w, block[4 * e + 1]);
        block[4 * e + 2] = fmaf(x.z, w, block[4 * e + 2]);
        block[4 * e + 3] = fmaf(x.w, w, block[4 * e + 3]);
      }
    }
    __syncthreads();
    if ((k0 - first) % 256 == 256 - kStep) {
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        folded[e] += block[e];
        block[e] = 0.f;
      }
    }
  }
  if (!again) return;
  float* out = parts_out(g, first_token, col);
  const long long ldo = g.shared ? g.n : g.ldo;
  const float bias = g.bias && !g.shared ? g.bias[col] : 0.f;
#pragma unroll
  for (int e = 0; e < 32; ++e)
    if (again >> e & 1u) out[e * ldo] = (folded[e] + block[e]) + bias;
}

__global__ void __launch_bounds__(kPartThreads, 1) gemm_parts_kernel(const __grid_constant__ PartsArgs g) {
  extern __shared__ unsigned char parts_smem[];
  __shared__ __align__(8) unsigned long long bars[1];
  __shared__ uint32_t tmem_address;
  __shared__ uint32_t odd[2][4], nan[2][4];        // rows of W and of A, a bit each: with a value that has no parts; with a NaN
  const uint32_t tiles = (smem_address(parts_smem) + 1023u) & ~1023u;
  const uint32_t bar = smem_address(bars);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = (int)blockIdx.y * kPartRows, col0 = (int)blockIdx.x * kPartRows;
  const int blocks = (g.k + kPartK - 1) / kPartK, first = (int)blockIdx.z * g.blocks_each, last = min(blocks, first + g.blocks_each);
  if (tid < 8) (&odd[0][0])[tid] = (&nan[0][0])[tid] = 0u;
  if (tid == 0) {
    bar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_address(&tmem_address)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_address;
  pdl_launch_dependents();
  pdl_wait();
  // this thread brings eight columns of rows 64 apart, two of either operand
  const int chunk = tid & 7, first_row = tid >> 3;
  float4 w_next[2][2], a_next[2][2];
  auto fetch = [&](int block) {
    const int at = block * kPartK + chunk * 8;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int wr = col0 + first_row + 64 * i, ar = row0 + first_row + 64 * i;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4* from = reinterpret_cast<const float4*>(g.w + (long long)wr * g.k + at);
      const bool there = wr < g.n && at < g.k;                    // k is a multiple of eight
      w_next[i][0] = there ? __ldg(from) : zero;
      w_next[i][1] = there ? __ldg(from + 1) : zero;
      const float4* rows = reinterpret_cast<const float4*>(g.a + (long long)ar * g.lda + at);
      const bool in = ar < g.m && at < g.k;
      a_next[i][0] = in ? rows[0] : zero;
      a_next[i][1] = in ? rows[1] : zero;
    }
  };
  bool ended = true;
  uint32_t marks = 0;                              // which of this thread's four rows (W, A, W, A) had a value without parts
  auto store = [&](uint32_t stage) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = first_row + 64 * i;
      const uint32_t at = stage + row * 128 + ((chunk ^ (row & 7)) << 4);
      uint4 part[3];
      marks |= split_eight(w_next[i][0], w_next[i][1], part) ? 0u : 1u << (2 * i);
#pragma unroll
      for (int j = 0; j < 3; ++j)
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + j * kPartTile), "r"(part[j].x), "r"(part[j].y), "r"(part[j].z), "r"(part[j].w) : "memory");
      marks |= split_eight(a_next[i][0], a_next[i][1], part) ? 0u : 2u << (2 * i);
#pragma unroll
      for (int j = 0; j < 3; ++j)
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + (3 + j) * kPartTile), "r"(part[j].x), "r"(part[j].y), "r"(part[j].z), "r"(part[j].w) : "memory");
    }
  };
  // D = F32, A = B = BF16, both K-major, N = 128, M = 128
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kPartRows >> 3) << 17) | ((uint32_t)(kPartRows >> 4) << 24);
  // this thread's 32 outputs: row col0 + 32 (warp & 3) + lane of W with 32 rows of A
  float sums[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) sums[e] = 0.f;
  const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 32), total = mine + 256;
  // the sums of the i-th block of this CTA: of its first 32 columns, and of the others
  auto promote = [&](int i) {
    ended = bar_poll(bar, i & 1) && ended;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int part = 0; part < 4; ++part) {
      float v[16];
      tmem_ld16(mine + (part & 1) * 128 + (part >> 1) * 16, v);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) sums[(part >> 1) * 16 + e] += v[e];
    }
    if (i % kPartFold == kPartFold - 1) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (i >= kPartFold) {
          float v[16];
          tmem_ld16(total + half * 16, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) sums[half * 16 + e] += v[e];
        }
        uint32_t r[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(sums[half * 16 + e]);
        tmem_st16(total + half * 16, r);
#pragma unroll
        for (int e = 0; e < 16; ++e) sums[half * 16 + e] = 0.f;
      }
      tmem_st_wait();
    }
  };
  const int count = last - first;
  if (count > 0) fetch(first);
  for (int i = 0; i < count; ++i) {
    const uint32_t stage = tiles + (i & 1) * kPartStage;
    store(stage);                       // its products of two blocks ago are over: their sums have been added
    if (i + 1 < count) fetch(first + i + 1);
    if (i > 0) promote(i - 1);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t w0 = desc_k_major(stage), a0 = desc_k_major(stage + 3 * kPartTile);
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int order = 2; order >= 0; --order)
#pragma unroll
          for (int p = 0; p <= order; ++p)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              const uint32_t step = (half * 2 + kk) * 32;
              mma_ss(tmem + half * 128, desc_advance(w0, p * kPartTile + step), desc_advance(a0, (order - p) * kPartTile + step),
                     kIdesc, order < 2 || p > 0 || kk > 0);
            }
      mma_commit(bar);
    }
    __syncwarp();
  }
  if (count > 0) promote(count - 1);
  if (count >= kPartFold) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float v[16];
      tmem_ld16(total + half * 16, v);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) sums[half * 16 + e] += v[e];
    }
  }
  if (marks) parts_mark(g, marks, row0 + first_row, col0 + first_row, first * kPartK + chunk * 8, min(g.k, last * kPartK), &odd[0][0], &nan[0][0]);
  const bool all_ended = __syncthreads_and(ended);            // and every mark is there
  if (!all_ended && tid == 0 && g.status) atomicOr(g.status, kStatusWaitExpired);
  const int col = col0 + (warp & 3) * 32 + lane, first_token = row0 + (warp >> 2) * 32;
  const int real = col < g.n ? max(0, min(32, g.m - first_token)) : 0;
  // this thread's outputs that its sums are not good for
  uint32_t again = odd[0][warp & 3] >> lane & 1u ? ~0u : odd[1][warp >> 2];
  float zero[4] = {};
#pragma unroll
  for (int e = 0; e < 32; ++e) zero[e & 3] = fmaf(sums[e], 0.f, zero[e & 3]);
  if ((zero[0] + zero[1]) + (zero[2] + zero[3]) != 0.f) {
#pragma unroll
    for (int e = 0; e < 32; ++e) again |= (fabsf(sums[e]) < INFINITY ? 0u : 1u) << e;
  }
  again &= nan[0][warp & 3] >> lane & 1u ? 0u : ~nan[1][warp >> 2];
  again = all_ended && real > 0 ? again & (~0u >> (32 - real)) : 0u;
  float* out = parts_out(g, first_token, col);
  const long long ldo = g.shared ? g.n : g.ldo;
  const float bias = real > 0 && g.bias && !g.shared ? g.bias[col] : 0.f;
  const uint32_t good = real == 32 ? ~again : ((1u << real) - 1u) & ~again;
  if (!all_ended) sums[0] = __int_as_float(0x7fffffff);
#pragma unroll
  for (int e = 0; e < 32; ++e)
    if (good >> e & 1u) out[e * ldo] = (all_ended ? sums[e] : sums[0]) + bias;
  if (__syncthreads_or(again != 0u))
    parts_by_fma(g, reinterpret_cast<float*>(parts_smem + (tiles - smem_address(parts_smem))), row0, col0, first * kPartK,
                 min(g.k, last * kPartK), again);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// The shares' sums, four and four in the order of K (one after the other, sixteen shares of uniform terms, K = 4,864, had an error of
// 0.874e-7 where FMA has 0.865e-7), and bias: four columns a thread where rows are whole groups of four (545 x 896 by four
// shares: 8.8 us with a thread and a 64-bit division an element).
template <int VEC>
__global__ void __launch_bounds__(256) gemm_parts_sum_kernel(const __grid_constant__ PartsArgs g, const float* sums, int shares) {
  pdl_launch_dependents();
  const long long total = (long long)g.m * g.n;
  const unsigned pieces = (unsigned)(g.n / VEC);
  const unsigned i = blockIdx.x * 256u + threadIdx.x;               // below 2^31 by the launch
  const unsigned r = i / pieces, c = (i - r * pieces) * VEC;
  pdl_wait();
  if (r >= (unsigned)g.m) return;
  const float* from = sums + (long long)r * g.n + c;
  float sum[VEC] = {};
  for (int s0 = 0; s0 < shares; s0 += 4) {
    float v[4][VEC];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float* at = from + (long long)min(s0 + s, shares - 1) * total;
      if constexpr (VEC == 4) {
        const float4 x = *reinterpret_cast<const float4*>(at);
        v[s][0] = x.x; v[s][1] = x.y; v[s][2] = x.z; v[s][3] = x.w;
      } else {
        v[s][0] = *at;
      }
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      sum[e] += (v[0][e] + (s0 + 1 < shares ? v[1][e] : 0.f)) + ((s0 + 2 < shares ? v[2][e] : 0.f) + (s0 + 3 < shares ? v[3][e] : 0.f));
  }
  float* out = g.out + (long long)r * g.ldo + c;
#pragma unroll
  for (int e = 0; e < VEC; ++e) sum[e] = g.bias ? sum[e] + g.bias[c + e] : sum[e];
  if constexpr (VEC == 4) *reinterpret_cast<float4*>(out) = make_float4(sum[0], sum[1], sum[2], sum[3]);
  else *out = sum[0];
}

}  // namespace einf

using namespace einf;

// sums: [shares][m][n] floats where shares (up to 16) is more than one.
extern "C" int einf_gemm_parts(const float* a, const float* w, const float* bias, float* out, int m, int n, int k, long long lda,
                               long long ldo, int shares, float* sums, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  const int blocks = (k + kPartK - 1) / kPartK;
  if (k <= 0 || k % 8 || lda % 4 || ((uintptr_t)a & 15) || ((uintptr_t)w & 15) || shares < 1 || shares > 16 || shares > blocks ||
      (shares > 1 && !sums) || (m + kPartRows - 1) / kPartRows > 65535)
    return (int)cudaErrorInvalidValue;
  PartsArgs g{a, w, bias, shares > 1 ? sums : out, m, n, k, lda, ldo, (blocks + shares - 1) / shares, shares > 1, status};
  cudaError_t e = cudaFuncSetAttribute(gemm_parts_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPartSmem);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid((n + kPartRows - 1) / kPartRows, (m + kPartRows - 1) / kPartRows, shares);
  e = launch_pdl(gemm_parts_kernel, grid, dim3(kPartThreads), kPartSmem, stream, g);
  if (e != cudaSuccess || shares == 1) return (int)e;
  g.out = out;
  const bool quads = n % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)sums & 15) == 0;
  const long long ctas = ((long long)m * n / (quads ? 4 : 1) + 255) / 256;
  if (ctas >= 1ll << 23) return (int)cudaErrorInvalidValue;        // the sums would be larger than the caller shares K for
  return (int)launch_pdl(quads ? gemm_parts_sum_kernel<4> : gemm_parts_sum_kernel<1>, dim3((unsigned)ctas), dim3(256), 0, stream, g,
                         (const float*)sums, shares);
}
