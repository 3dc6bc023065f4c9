// The products of a layer for a handful of tokens (a decode step of up to 16 requests), each with what stands
// before and behind it in one launch: the norm of the residual stream in front of the QKV and the gate/up product;
// bias, rotation and the cache write behind QKV; the addition to the residual stream behind the attention's output
// product; SiLU and the product of the two branches behind gate/up.
//
// Such a step is bound by the length of its chain, not by its bytes: at 0.5B sizes a layer moves 30 MB, 4.6 us worth,
// and took 24.4 us for one token and 29.0 for eight (contexts of 1,024 and 4,096, attention 4.4 and 7.8 of it) as nine
// launches; as these four and the attention it takes 17.6 and 22.8 (QKV 2.5 / 3.2, output 2.0 / 2.4, gate/up 4.1 / 4.2, down
// 2.8 / 3.8).  So every kernel here has its weights on the way to shared memory before it waits for the kernel in front of
// it (one bulk copy a row), and behind that wait one or two round trips to L2, one chain of a few matrix instructions, one
// meeting of the CTA's warps and the stores.  No partial sums leave a CTA: its warps share K.
//
// The tokens are the sixteen rows of mma.sync m16n8k16 (eight of them zero for up to eight tokens), eight weight
// rows its columns.  Both operands are taken in the same order of K within 32 elements, so that a lane's operands of
// two instructions are 16 consecutive bytes of a row; weight rows lie 64 bytes beyond a multiple of 128 apart, which puts
// the eight lanes of a quarter of such a load on all 32 banks.  No warp reads an activation that another warp of the
// CTA reads, so activations come straight from L2 into registers.  The norm's factor 1 / rms is a number per token: the
// product runs on bf16(weight * h), the squares are added up on the way and the sums are multiplied behind the product.
//
// Gate/up takes 32 rows and four warps a CTA: many small CTAs load while others compute (eight warps 4.6 to 5.9 us,
// 16 rows 4.4 to 7.5, 64 rows 7.3 to 8.0, one wave of persistent CTAs with a ring of rows 6.2; a prefetch of the
// later matrices into L2 by the earlier kernels gained nothing).  Rows above 1,024 elements keep the separate kernels:
// at 1.5B sizes (94 MB a layer, gate/up 11.5 us) a layer takes 34.9 and 45.0 us here and 34.2 and 40.3 there.
#include "mma_sync.cuh"
#include "tcgen05.cuh"

namespace einf {

enum FewEnd : int { kFewQkv = 0, kFewSilu = 1, kFewAdd = 2, kFewStore = 3 };

struct FewArgs {
  const __nv_bfloat16* weight;   // [rows, k]
  int k, rows, tokens;
  // in front: the stream and what is pending (may be null), normalised; or rows as they are
  const float* residual;         // [tokens, k]
  const float* pending;          // [tokens, k]
  const float* norm_weight;      // [k]
  float eps;
  const __nv_bfloat16* x;        // [tokens, k]
  // behind
  const float* bias;             // QKV: [rows] or null
  const int* positions;
  const float* inv_freq;
  const int* slots;              // null: keys and values are not stored
  __nv_bfloat16* q_out;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  int num_heads, num_kv_heads, head_size, rotary, page_size, num_pages;
  __nv_bfloat16* out;            // SiLU: [tokens, rows / 2]
  float* sum;                    // add: the stream [tokens, rows]; store: [tokens, rows]
  const float* add;              // add: pending (may be null)
  int* status;
};

__host__ __device__ constexpr int few_row_bytes(int k) { return ((k * 2 + 127) & ~127) + 64; }

// RT: groups of eight weight rows a CTA; WARPS share K, 32 elements at a time in turn; BATCH: such pieces of a warp in flight;
// HI: more than eight tokens; NORM: what is in front.
template <int RT, int WARPS, int BATCH, bool HI, bool NORM, int END>
__global__ void __launch_bounds__(WARPS * 32) few_tokens_kernel(FewArgs a) {
  pdl_launch_dependents();
  constexpr int kRows = RT * 8, kTokens = HI ? 16 : 8, kPitch = kTokens + 1;
  extern __shared__ __align__(128) unsigned char few_smem[];
  __shared__ float red[WARPS * kRows * kPitch];
  __shared__ float squares[WARPS * kTokens];
  __shared__ __align__(8) unsigned long long arrived;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int tile = blockIdx.x, row_bytes = few_row_bytes(a.k);
  const uint32_t weights = smem_address(few_smem), norm = weights + kRows * row_bytes, bar = smem_address(&arrived);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (warp == 0) {
    if (lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kRows * a.k * 2 + (NORM ? a.k * 4 : 0)) : "memory");
    __syncwarp();
    for (int r = lane; r < kRows; r += 32) {
      int row;
      if (END == kFewQkv) {
        // half of the rows from either half of a head: both members of the pairs that turn together
        const int tiles = a.head_size / kRows, head = tile / tiles, part = tile - head * tiles;
        row = head * a.head_size + part * (kRows / 2) + (r < kRows / 2 ? r : r - kRows / 2 + a.head_size / 2);
      } else if (END == kFewSilu) {
        row = tile * (kRows / 2) + (r < kRows / 2 ? r : r - kRows / 2 + a.rows / 2);   // gate rows, and their up rows
      } else {
        row = tile * kRows + r;
      }
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(weights + r * row_bytes),
                   "l"(a.weight + (size_t)row * a.k), "r"(a.k * 2), "r"(bar)
                   : "memory");
    }
    if (NORM && lane == 0)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(norm), "l"(a.norm_weight),
                   "r"(a.k * 4), "r"(bar)
                   : "memory");
  }
  // what the end needs of the step's inputs and of the bias, before the wait as well
  constexpr int kEach = END == kFewQkv || END == kFewSilu ? kRows / 2 : kRows;     // outputs a token
  static_assert(END == kFewSilu || kEach * kTokens <= WARPS * 32, "a thread has one result");
  int item = tid % kEach, token = tid / kEach;
  const bool ends = token < a.tokens;
  int head = 0, dim = 0, slot = -1;
  bool is_v = false;
  float cosine = 1.f, sine = 0.f, bias_a = 0.f, bias_b = 0.f;
  if (END == kFewQkv && ends) {
    const int tiles = a.head_size / kRows;
    head = tile / tiles;
    dim = (tile - head * tiles) * kEach + item;
    is_v = head >= a.num_heads + a.num_kv_heads;
    if (!is_v && a.rotary) sincosf((float)a.positions[token] * a.inv_freq[dim], &sine, &cosine);
    if (a.bias) {
      bias_a = a.bias[head * a.head_size + dim];
      bias_b = a.bias[head * a.head_size + dim + a.head_size / 2];
    }
    if (a.slots) slot = a.slots[token];
  }
  pdl_wait();
  float before = 0.f;                      // of the stream, where this thread's sum goes
  if (END == kFewAdd && ends) {
    const size_t at = (size_t)token * a.rows + tile * kRows + item;
    before = a.sum[at];
    if (a.add) before += a.add[at];
  }
  float acc[RT][4] = {};
  float low = 0.f, high = 0.f;
  const int pieces = a.k >> 5;
  bool there = false, failed = false;
  for (int base = warp; base < pieces; base += WARPS * BATCH) {
    uint4 xa[BATCH], xb[HI ? BATCH : 1];
    if (NORM) {
      float4 h[BATCH][HI ? 4 : 2];
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int at = (base + u * WARPS) * 32 + t * 8;
        const bool in = base + u * WARPS < pieces;
#pragma unroll
        for (int half = 0; half < (HI ? 2 : 1); ++half) {
          const bool real = in && g + half * 8 < a.tokens;
          const float4* from = reinterpret_cast<const float4*>(a.residual + (size_t)(g + half * 8) * a.k + at);
          h[u][half * 2] = real ? from[0] : make_float4(0.f, 0.f, 0.f, 0.f);
          h[u][half * 2 + 1] = real ? from[1] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      if (END == kFewQkv && a.pending) {
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
          const int at = (base + u * WARPS) * 32 + t * 8;
          const bool in = base + u * WARPS < pieces;
#pragma unroll
          for (int half = 0; half < (HI ? 2 : 1); ++half) {
            if (!(in && g + half * 8 < a.tokens)) continue;
            const float4* from = reinterpret_cast<const float4*>(a.pending + (size_t)(g + half * 8) * a.k + at);
            const float4 p = from[0], r = from[1];
            float4 &v = h[u][half * 2], &w = h[u][half * 2 + 1];
            v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
            w.x += r.x; w.y += r.y; w.z += r.z; w.w += r.w;
          }
        }
      }
      if (!there) failed = !bar_poll(bar, 0);
      there = true;
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int at = (base + u * WARPS) * 32 + t * 8;
        if (base + u * WARPS >= pieces) break;
        float4 n0, n1;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(n0.x), "=f"(n0.y), "=f"(n0.z), "=f"(n0.w) : "r"(norm + at * 4) : "memory");
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(n1.x), "=f"(n1.y), "=f"(n1.z), "=f"(n1.w) : "r"(norm + at * 4 + 16) : "memory");
#pragma unroll
        for (int half = 0; half < (HI ? 2 : 1); ++half) {
          const float4 v = h[u][half * 2], w = h[u][half * 2 + 1];
          float& squared = half ? high : low;
          squared += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w + w.x * w.x + w.y * w.y + w.z * w.z + w.w * w.w;
          (half ? xb[HI ? u : 0] : xa[u]) = make_uint4(pack_pair(v.x * n0.x, v.y * n0.y), pack_pair(v.z * n0.z, v.w * n0.w),
                                                       pack_pair(w.x * n1.x, w.y * n1.y), pack_pair(w.z * n1.z, w.w * n1.w));
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int at = (base + u * WARPS) * 32 + t * 8;
        const bool in = base + u * WARPS < pieces;
        xa[u] = in && g < a.tokens ? *reinterpret_cast<const uint4*>(a.x + (size_t)g * a.k + at) : make_uint4(0u, 0u, 0u, 0u);
        if (HI) xb[u] = in && g + 8 < a.tokens ? *reinterpret_cast<const uint4*>(a.x + (size_t)(g + 8) * a.k + at) : make_uint4(0u, 0u, 0u, 0u);
      }
      if (!there) failed = !bar_poll(bar, 0);
      there = true;
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      if (base + u * WARPS >= pieces) break;
      const uint4 hi = HI ? xb[HI ? u : 0] : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t first[4] = {xa[u].x, hi.x, xa[u].y, hi.y}, second[4] = {xa[u].z, hi.z, xa[u].w, hi.w};
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        uint4 w;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                     : "r"(weights + (r * 8 + g) * row_bytes + (base + u * WARPS) * 64 + t * 16)
                     : "memory");
        mma_bf16_16816(acc[r], first, w.x, w.y);
        mma_bf16_16816(acc[r], second, w.z, w.w);
      }
    }
  }
  if (!there) failed = !bar_poll(bar, 0);     // a warp without a piece: no CTA ends with a copy under way
  if (failed) atomicOr(a.status, kStatusWaitExpired);
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    float* to = red + (warp * kRows + r * 8 + 2 * t) * kPitch + g;
    to[0] = acc[r][0];
    to[kPitch] = acc[r][1];
    if (HI) {
      to[8] = acc[r][2];
      to[kPitch + 8] = acc[r][3];
    }
  }
  if (NORM) {
    low += __shfl_xor_sync(0xffffffffu, low, 1);
    low += __shfl_xor_sync(0xffffffffu, low, 2);
    if (t == 0) squares[warp * kTokens + g] = low;
    if (HI) {
      high += __shfl_xor_sync(0xffffffffu, high, 1);
      high += __shfl_xor_sync(0xffffffffu, high, 2);
      if (t == 0) squares[warp * kTokens + g + 8] = high;
    }
  }
  __syncthreads();
  for (; token < a.tokens; token += WARPS * 32 / kEach) {
    float one = 0.f, two = 0.f, scale = 1.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      one += red[(w * kRows + item) * kPitch + token];
      if (END == kFewQkv || END == kFewSilu) two += red[(w * kRows + kEach + item) * kPitch + token];
    }
    if (NORM) {
      float total = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) total += squares[w * kTokens + token];
      scale = rsqrtf(total / (float)a.k + a.eps);
      one *= scale;
      two *= scale;
    }
    if (END == kFewQkv) {
      one += bias_a;
      two += bias_b;
      __nv_bfloat16* to;
      if (head < a.num_heads) {
        to = a.q_out + ((size_t)token * a.num_heads + head) * a.head_size;
      } else {
        if (slot < 0) continue;
        const int page = slot / a.page_size, offset = slot - page * a.page_size;
        if (page >= a.num_pages) {
          atomicOr(a.status, kStatusBadPage);
          continue;
        }
        const int kv = is_v ? head - a.num_heads - a.num_kv_heads : head - a.num_heads;
        to = (is_v ? a.v_cache : a.k_cache) + (((size_t)page * a.num_kv_heads + kv) * a.page_size + offset) * a.head_size;
      }
      const bool turns = !is_v && a.rotary;     // else the halves do not meet: zero times infinity would not be zero
      to[dim] = __float2bfloat16_rn(turns ? one * cosine - two * sine : one);
      to[dim + a.head_size / 2] = __float2bfloat16_rn(turns ? two * cosine + one * sine : two);
    } else if (END == kFewSilu) {
      a.out[(size_t)token * (a.rows / 2) + tile * kEach + item] = __float2bfloat16_rn(one / (1.f + expf(-one)) * two);
    } else {
      const size_t at = (size_t)token * a.rows + tile * kRows + item;
      a.sum[at] = END == kFewAdd ? before + one : one;
    }
  }
}

template <int RT, int WARPS, int LOW_BATCH, int HIGH_BATCH, bool NORM, int END>
int few_launch(const FewArgs& a, cudaStream_t stream) {
  constexpr int kRows = RT * 8;
  const size_t smem = (size_t)kRows * few_row_bytes(a.k) + (NORM ? (size_t)a.k * 4 : 0);
  auto kernel = a.tokens > 8 ? few_tokens_kernel<RT, WARPS, HIGH_BATCH, true, NORM, END>
                             : few_tokens_kernel<RT, WARPS, LOW_BATCH, false, NORM, END>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_pdl(kernel, a.rows / kRows, WARPS * 32, smem, stream, a);
}

inline bool few_fits(int tokens, int k, const void* weight, int rows_a_cta, bool norm) {
  return tokens >= 1 && tokens <= 16 && k >= 32 && k % 32 == 0 && ((uintptr_t)weight & 15) == 0 &&
         (size_t)rows_a_cta * few_row_bytes(k) + (norm ? (size_t)k * 4 : 0) <= 200 * 1024;
}

}  // namespace einf

using namespace einf;

extern "C" int einf_few_qkv(const float* residual, const float* pending, const float* norm_weight, float eps, const void* weight,
                            const float* bias, const int* positions, const float* inv_freq, const int* slots, void* q_out,
                            void* k_cache, void* v_cache, int tokens, int k, int num_heads, int num_kv_heads, int head_size,
                            int rotary, int page_size, int num_pages, int* status, cudaStream_t stream) {
  if (!few_fits(tokens, k, weight, 8, true) || head_size % 8 || ((uintptr_t)residual & 15) || ((uintptr_t)pending & 15) ||
      ((uintptr_t)norm_weight & 15) || (slots && page_size <= 0))
    return (int)cudaErrorInvalidValue;
  FewArgs a = {};
  a.weight = (const __nv_bfloat16*)weight;
  a.k = k;
  a.rows = (num_heads + 2 * num_kv_heads) * head_size;
  a.tokens = tokens;
  a.residual = residual;
  a.pending = pending;
  a.norm_weight = norm_weight;
  a.eps = eps;
  a.bias = bias;
  a.positions = positions;
  a.inv_freq = inv_freq;
  a.slots = slots;
  a.q_out = (__nv_bfloat16*)q_out;
  a.k_cache = (__nv_bfloat16*)k_cache;
  a.v_cache = (__nv_bfloat16*)v_cache;
  a.num_heads = num_heads;
  a.num_kv_heads = num_kv_heads;
  a.head_size = head_size;
  a.rotary = rotary;
  a.page_size = page_size;
  a.num_pages = num_pages;
  a.status = status;
  return few_launch<1, 8, 4, 4, true, kFewQkv>(a, stream);
}

extern "C" int einf_few_gate_up(const float* residual, const float* norm_weight, float eps, const void* weight, void* out, int tokens,
                                int k, int intermediate, int* status, cudaStream_t stream) {
  if (!few_fits(tokens, k, weight, 32, true) || intermediate % 16 || ((uintptr_t)residual & 15) || ((uintptr_t)norm_weight & 15))
    return (int)cudaErrorInvalidValue;
  FewArgs a = {};
  a.weight = (const __nv_bfloat16*)weight;
  a.k = k;
  a.rows = 2 * intermediate;
  a.tokens = tokens;
  a.residual = residual;
  a.norm_weight = norm_weight;
  a.eps = eps;
  a.out = (__nv_bfloat16*)out;
  a.status = status;
  return few_launch<4, 4, 4, 4, true, kFewSilu>(a, stream);
}

// add_to_stream: out += pending + x weight^T (pending may be null); else out = x weight^T.
extern "C" int einf_few_product(const void* x, const void* weight, const float* pending, float* out, int add_to_stream, int tokens,
                                int k, int rows, int* status, cudaStream_t stream) {
  if (!few_fits(tokens, k, weight, 8, false) || rows % 8 || ((uintptr_t)x & 15)) return (int)cudaErrorInvalidValue;
  FewArgs a = {};
  a.weight = (const __nv_bfloat16*)weight;
  a.k = k;
  a.rows = rows;
  a.tokens = tokens;
  a.x = (const __nv_bfloat16*)x;
  a.sum = out;
  a.add = pending;
  a.status = status;
  // sixteen warps share a long K, eight a short one (12 or 20 warps for 4,864: 3.8 and 3.9 against 2.8 us)
  if (k > 2048)
    return add_to_stream ? few_launch<1, 16, 10, 5, false, kFewAdd>(a, stream) : few_launch<1, 16, 10, 5, false, kFewStore>(a, stream);
  return add_to_stream ? few_launch<1, 8, 4, 4, false, kFewAdd>(a, stream) : few_launch<1, 8, 4, 4, false, kFewStore>(a, stream);
}
