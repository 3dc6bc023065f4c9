// out[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) with 32-bit FMA accumulation on the
// CUDA cores: the product for operands of mixed type (bfloat16 activations against a
// matrix the checkpoint stores in 32-bit) and for 32-bit rows that are not whole
// aligned groups of four (gemm_parts.cu has the others).  Any M, N, K.
// Sums over K are blocked: every 256 terms the running sum is folded into a second
// accumulator, so that the rounding of a long sum (K of 18,944 in a 7B-size down
// projection) grows like the root of the block plus the root of the number of blocks and
// not like the root of K.  The order of additions depends on K alone.
//
// Bound by FMA (70 TFLOP/s measured over the GPU) and, next to it, by shared memory: an SM multiplies 128 and reads 32
// operands a cycle, so a thread has 8 x 8 outputs (4 x 4, as before, spends twice as long on its reads as on its FMAs).  A
// CTA has 64 x 128 outputs; the next 16 columns of both operands are on their way in registers while this tile is
// multiplied out of shared memory.  The FMAs are taken in pairs along the columns, each rounded as one.  Where such
// tiles are too few for the GPU (the down and output projections of a few hundred tokens, every product of a few),
// CTAs share K, whole blocks of 256 terms each, leave every block's sum in a workspace, and a second kernel adds the
// blocks up in order: the result is the same bit for bit however many share.
//
// Measured (B200, us, with a thread of 4 x 4 before): 545 rows, 896 -> 1,152 99 -> 40, 896 -> 896 60 -> 41, 896 -> 9,728 424 ->
// 211, 4,864 -> 896 312 -> 117; 2,048 rows, 3,584 -> 4,608 2,690 -> 1,300 (52 TFLOP/s); one row, 896 -> 9,728 82 -> 40.
// Tried: a thread of 8 x 4 in 64 x 64 tiles, 43 TFLOP/s at the largest of these; the rows' operand twice in shared memory
// in the place of moves into pairs, 31; sums of a cluster's CTAs in shared memory instead of the workspace, 185 us at
// 4,864 -> 896 (their room leaves two CTAs an SM).
//
// The reference's 32-bit path is F.linear through cuBLAS with TF32 off
// (src/einf/executors/torch/packed_qkv.py:148, qwen.py:207-208,489,773).
#include "common.cuh"

namespace einf {

constexpr int kRows = 64, kCols = 128;  // rows of A and rows of W per CTA
constexpr int kTileK = 16;
constexpr int kThreads = 128;           // 8 x 16, 8 x 8 outputs each
constexpr int kRowPitch = kRows + 4, kColPitch = kCols + 4;
constexpr int kBlock = 256;             // terms of a block sum

struct SimtArgs {
  const void* a; const void* w; const float* bias; void* out;
  float* block_sums;                    // [blocks of K][m][n], where CTAs share K
  int m, n, k;
  long long lda, ldo;
  int a_wide, w_wide;                   // rows in whole aligned groups of four elements
  int blocks_each;                      // blocks of 256 terms that a CTA takes
};

template <typename T>
__device__ __forceinline__ float4 load_four(const T* row, int kk, int k, bool wide) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!row || kk >= k) return v;
  if (wide) {                           // k is a multiple of four
    if constexpr (sizeof(T) == 4) {
      v = *reinterpret_cast<const float4*>(row + kk);
    } else {
      const uint2 raw = *reinterpret_cast<const uint2*>(row + kk);
      v.x = __uint_as_float(raw.x << 16);
      v.y = __uint_as_float(raw.x & 0xffff0000u);
      v.z = __uint_as_float(raw.y << 16);
      v.w = __uint_as_float(raw.y & 0xffff0000u);
    }
    return v;
  }
  v.x = to_float(row[kk]);
  if (kk + 1 < k) v.y = to_float(row[kk + 1]);
  if (kk + 2 < k) v.z = to_float(row[kk + 2]);
  if (kk + 3 < k) v.w = to_float(row[kk + 3]);
  return v;
}

__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
// two 32-bit FMAs in one instruction, each rounded as fmaf rounds it
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t x, uint64_t y) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y));
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

// kShared: the CTAs along z share K (blocks_each blocks each).
template <typename TA, typename TW, typename TOut, bool kShared>
__global__ void __launch_bounds__(kThreads, 3)
gemm_simt_kernel(const __grid_constant__ SimtArgs g) {
  __shared__ __align__(16) float a_s[2][kTileK][kRowPitch];
  __shared__ __align__(16) float w_s[2][kTileK][kColPitch];
  extern __shared__ __align__(16) float4 totals[];         // the running totals, every thread's own 16 quadruples
  pdl_launch_dependents();
  pdl_wait();
  const int col0 = (int)blockIdx.x * kCols, row0 = (int)blockIdx.y * kRows;
  const int first_block = kShared ? (int)blockIdx.z * g.blocks_each : 0;
  const int k_begin = first_block * kBlock;
  const int k_end = kShared ? min(g.k, k_begin + g.blocks_each * kBlock) : g.k;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // what this thread brings: four columns of two rows of A and of four rows of W, 32 rows apart (lanes
  // four to a row: eight to a column, so that a quarter of a warp reads eight rows, measured 342 us where this takes 254)
  const int load_row = threadIdx.x >> 2, load_k = (threadIdx.x & 3) * 4;
  const TA* a_rows[2];
  const TW* w_rows[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = row0 + load_row + 32 * i;
    a_rows[i] = row < g.m ? (const TA*)g.a + (long long)row * g.lda : nullptr;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = col0 + load_row + 32 * i;
    w_rows[i] = row < g.n ? (const TW*)g.w + (long long)row * g.k : nullptr;
  }
  float4 a_next[2], w_next[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) a_next[i] = load_four(a_rows[i], k0 + load_k, k_end, g.a_wide);
#pragma unroll
    for (int i = 0; i < 4; ++i) w_next[i] = load_four(w_rows[i], k0 + load_k, k_end, g.w_wide);
  };
  auto stash = [&](int buffer) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a_s[buffer][load_k][load_row + 32 * i] = a_next[i].x;
      a_s[buffer][load_k + 1][load_row + 32 * i] = a_next[i].y;
      a_s[buffer][load_k + 2][load_row + 32 * i] = a_next[i].z;
      a_s[buffer][load_k + 3][load_row + 32 * i] = a_next[i].w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w_s[buffer][load_k][load_row + 32 * i] = w_next[i].x;
      w_s[buffer][load_k + 1][load_row + 32 * i] = w_next[i].y;
      w_s[buffer][load_k + 2][load_row + 32 * i] = w_next[i].z;
      w_s[buffer][load_k + 3][load_row + 32 * i] = w_next[i].w;
    }
  };
  // a warp has 32 rows x 64 columns: lanes four along the rows, eight along the columns (two groups of four
  // columns, 32 apart)
  const int ty = (warp >> 1) * 32 + (lane >> 3) * 8, tx = (warp & 1) * 64 + (lane & 7) * 4;
  uint64_t acc[8][4];                              // columns in pairs
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

  int block = 0;
  if (k_begin < k_end) {
    fetch(k_begin);
    stash(0);
  }
  __syncthreads();
  int buffer = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += kTileK, buffer ^= 1) {
    const bool more = k0 + kTileK < k_end;
    if (more) fetch(k0 + kTileK);
#pragma unroll
    for (int kk = 0; kk < kTileK; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(&a_s[buffer][kk][ty]);
      const float4 a1 = *reinterpret_cast<const float4*>(&a_s[buffer][kk][ty + 4]);
      const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(&w_s[buffer][kk][tx]);
      const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(&w_s[buffer][kk][tx + 32]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t aa = pack2(av[i], av[i]);
        fma2(acc[i][0], aa, w0.x);
        fma2(acc[i][1], aa, w0.y);
        fma2(acc[i][2], aa, w1.x);
        fma2(acc[i][3], aa, w1.y);
      }
    }
    if (more) stash(buffer ^ 1);
    const bool full = ((k0 - k_begin) & (kBlock - 1)) == kBlock - kTileK;
    if (full || (kShared && !more)) {              // a block of 256 terms (or the last of K) is complete
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          const float2 x = unpack2(acc[i][j]), y = unpack2(acc[i][j + 1]);
          acc[i][j] = acc[i][j + 1] = 0ull;
          if constexpr (kShared) {
            const int r = row0 + ty + i, c = col0 + tx + 16 * j;
            float* to = g.block_sums + ((long long)(first_block + block) * g.m + r) * g.n + c;
            if (r >= g.m) continue;
            if (g.n % 4 == 0) {
              if (c < g.n) *reinterpret_cast<float4*>(to) = make_float4(x.x, x.y, y.x, y.y);
            } else {
              const float v[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (c + e < g.n) to[e] = v[e];
            }
          } else {
            float4* at = totals + (i * 2 + j / 2) * kThreads + threadIdx.x;
            float4 t = block ? *at : make_float4(0.f, 0.f, 0.f, 0.f);
            t.x += x.x;
            t.y += x.y;
            t.z += y.x;
            t.w += y.y;
            *at = t;
          }
        }
      ++block;
    }
    __syncthreads();
  }
  if constexpr (!kShared) {
    TOut* out = (TOut*)g.out;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = row0 + ty + i;
      if (r >= g.m) continue;
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const float4 t = block ? totals[(i * 2 + j / 2) * kThreads + threadIdx.x] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float2 x = unpack2(acc[i][j]), y = unpack2(acc[i][j + 1]);
        const float v[4] = {t.x + x.x, t.y + x.y, t.z + y.x, t.w + y.y};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = col0 + tx + 16 * j + e;
          if (c < g.n) out[(long long)r * g.ldo + c] = from_float<TOut>(g.bias ? v[e] + g.bias[c] : v[e]);
        }
      }
    }
  }
}

// The blocks' sums added up in the order of K, bias, the result's type.
template <typename TOut>
__global__ void __launch_bounds__(256)
gemm_simt_sum_kernel(const __grid_constant__ SimtArgs g) {
  pdl_launch_dependents();
  pdl_wait();
  const long long total = (long long)g.m * g.n;
  const int blocks = (g.k + kBlock - 1) / kBlock;
  TOut* out = (TOut*)g.out;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    float sum = 0.f;
    constexpr int kAtOnce = 8;
    for (int b0 = 0; b0 < blocks; b0 += kAtOnce) {
      float v[kAtOnce];
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u) v[u] = b0 + u < blocks ? g.block_sums[(b0 + u) * total + i] : 0.f;
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u)
        if (b0 + u < blocks) sum += v[u];
    }
    const int r = (int)(i / g.n), c = (int)(i - (long long)r * g.n);
    out[(long long)r * g.ldo + c] = from_float<TOut>(g.bias ? sum + g.bias[c] : sum);
  }
}

template <typename TA, typename TW, typename TOut>
static cudaError_t launch_simt(SimtArgs g, int share, cudaStream_t stream) {
  const int blocks = (g.k + kBlock - 1) / kBlock;
  g.blocks_each = (blocks + share - 1) / share;
  const dim3 grid((g.n + kCols - 1) / kCols, (g.m + kRows - 1) / kRows, share);
  if (share > 1) {
    cudaError_t e = launch_pdl(gemm_simt_kernel<TA, TW, TOut, true>, grid, dim3(kThreads), 0, stream, g);
    if (e != cudaSuccess) return e;
    const long long ctas = ((long long)g.m * g.n + 255) / 256;
    return launch_pdl(gemm_simt_sum_kernel<TOut>, dim3((unsigned)(ctas < 148 * 8 ? ctas : 148 * 8)), dim3(256), 0, stream, g);
  }
  auto kernel = gemm_simt_kernel<TA, TW, TOut, false>;
  constexpr int kBytes = kRows * kCols * (int)sizeof(float);
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return e;
  return launch_pdl(kernel, grid, dim3(kThreads), kBytes, stream, g);
}

}  // namespace einf

using namespace einf;

template <typename TA, typename TW>
static int launch(const SimtArgs& g, int share, int out_dtype, cudaStream_t stream) {
  if (out_dtype == kFloat32) return (int)launch_simt<TA, TW, float>(g, share, stream);
  return (int)launch_simt<TA, TW, __nv_bfloat16>(g, share, stream);
}

// How many CTAs share K, as far as the blocks' sums take no more than `limit` bytes.  CTAs run three an SM, but an SM's rate does
// not grow with them, so a launch takes as long as the SM with the most blocks of 256 terms: CTAs an SM, rounded up, times
// blocks a CTA.  Sharing costs three quarters of a block more (the workspace and the second kernel); of equal shares the
// larger one, whose CTAs hide one another's waits better.  Measured (us, alone / the rule): 63 tiles, K = 4,864 295 / 129; 81, K =
// 896 61 / 43; 200, K = 2,048 217 / 158; 288, K = 1,024 115 / alone (126 by two); 300, K = 896 136 / 118; 384, K = 1,024 160 / 164 (178
// by two); 440, K = 515 95 / alone (112 by two); 448, K = 1,024 207 / 190.
extern "C" int einf_gemm_simt_shares(int m, int n, int k, long long limit) {
  const long long tiles = (long long)((m + kRows - 1) / kRows) * ((n + kCols - 1) / kCols);
  const int blocks = (k + kBlock - 1) / kBlock;
  if (tiles <= 0 || 4ll * blocks * m * n > limit) return 1;
  constexpr int kSms = 148;
  int share = 1;
  long long best = 4 * ((tiles + kSms - 1) / kSms) * blocks;          // in quarters of a block
  const long long alone = best;
  for (int s = 2; s <= blocks; ++s) {
    const int each = (blocks + s - 1) / s;
    if ((blocks + each - 1) / each != s) continue;                    // no CTA without a block
    const long long cost = 4 * ((tiles * s + kSms - 1) / kSms) * each + 3;
    if (cost < alone && cost <= best) {
      best = cost;
      share = s;
    }
  }
  return share;
}

// lda / ldo: row strides of A and out in elements (rows of A may be a strided view).  block_sums: [blocks of 256
// terms of K][m][n] floats where `share` (einf_gemm_simt_shares) is more than one.
extern "C" int einf_gemm_simt(const void* a, int a_dtype, const void* w, int w_dtype, const float* bias,
                              void* out, int out_dtype, int m, int n, int k, long long lda,
                              long long ldo, int share, float* block_sums, cudaStream_t stream) {
  if (m == 0 || n == 0) return 0;
  if (share < 1 || share > 65535 || (share > 1 && !block_sums)) return (int)cudaErrorInvalidValue;
  const int a_size = a_dtype == kFloat32 ? 4 : 2, w_size = w_dtype == kFloat32 ? 4 : 2;
  SimtArgs g;
  g.a = a; g.w = w; g.bias = bias; g.out = out; g.block_sums = block_sums;
  g.m = m; g.n = n; g.k = k; g.lda = lda; g.ldo = ldo;
  g.a_wide = k % 4 == 0 && lda % 4 == 0 && (uintptr_t)a % (4 * a_size) == 0;
  g.w_wide = k % 4 == 0 && (uintptr_t)w % (4 * w_size) == 0;
  g.blocks_each = 0;
  if (a_dtype == kFloat32) {
    if (w_dtype == kFloat32) return launch<float, float>(g, share, out_dtype, stream);
    return launch<float, __nv_bfloat16>(g, share, out_dtype, stream);
  }
  if (w_dtype == kFloat32) return launch<__nv_bfloat16, float>(g, share, out_dtype, stream);
  return launch<__nv_bfloat16, __nv_bfloat16>(g, share, out_dtype, stream);
}
