// Warp-level matrix instructions (mma.sync m16n8k16, bfloat16 operands, 32-bit sums) and what feeds them, and 32-bit
// values as three bfloat16 parts.
//
// Measured on this part: 550 TFLOP/s over all multiprocessors from registers, against 70 TFLOP/s of 32-bit FMA, so a
// 32-bit operand may be taken as three bfloat16 parts (8 bits of the significand each, all 24 together) and
// three products, or six where both operands are 32-bit, and still be faster than FMA.
#pragma once

#include "common.cuh"

namespace einf {

__device__ __forceinline__ uint32_t smem_address(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void ldsm_x2_trans(uint32_t (&r)[2], uint32_t address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(address));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same with a sum that starts at zero.
__device__ __forceinline__ void mma_bf16_16816_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// acc += A B over 16 elements, operands given in PA and PB bfloat16 parts, largest first.  The instruction cuts its
// sums off where 32-bit FMA rounds them, so a long chain of it drifts: the products of the smaller parts come
// first, the product of the largest parts last, and the 16-element sum is added to the running one by a rounded
// addition.  (Chained without that, sums of 64 to 128 elements were three times as far from 64 bits as FMA.)
template <int PA, int PB>
__device__ __forceinline__ void mma_parts(float (&acc)[4], const uint32_t (&a)[PA][4], const uint32_t (&b)[PB][2]) {
  constexpr int kOrder = (PA > PB ? PA : PB) - 1;      // parts i and j count while i + j <= kOrder
  float t[4];
  bool first = true;
#pragma unroll
  for (int order = kOrder; order >= 0; --order)
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int j = order - i;
      if (j < 0 || j >= PB) continue;
      if (first) mma_bf16_16816_zero(t, a[i], b[j][0], b[j][1]);
      else mma_bf16_16816(t, a[i], b[j][0], b[j][1]);
      first = false;
    }
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] += t[e];
}

// Eight or sixteen bytes from global to shared memory in the background; `bytes` 0 writes zeros and reads nothing.
__device__ __forceinline__ void cp_async8(uint32_t smem, const void* gmem, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void sts_u32(uint32_t address, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(address), "r"(v) : "memory");
}
__device__ __forceinline__ void sts_v2(uint32_t address, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(address), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t address) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(address) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds_v2(uint32_t address) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(address) : "memory");
  return v;
}
__device__ __forceinline__ float low_bf16(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float high_bf16(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_pair(float low, float high) {
  __nv_bfloat162 v = __floats2bfloat162_rn(low, high);
  return *reinterpret_cast<uint32_t*>(&v);
}

// The halves of a pair of bfloat16 that are infinite or NaN, as their highest bits.
__device__ __forceinline__ uint32_t not_finite(uint32_t pair) { return ((pair & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }

// Byte of a 16-byte piece of a row whose rows are 128-byte lines: exchanged by the row's last three bits, so that the eight
// rows of an ldmatrix meet no bank twice.
__device__ __forceinline__ uint32_t swizzled(int row, int piece, int pitch) {
  return (uint32_t)(row * pitch + ((piece & ~7) | ((piece ^ row) & 7)) * 16);
}

// Which rows of a prompt a CTA of (row tiles x heads) has: pairs in the order of their keys, the last tiles first; every second
// wave of CTAs (`wave`: multiprocessors) takes them from the other end, so that an SM's CTAs, which all run at once, are
// long and short ones.
__device__ __forceinline__ void rows_of_cta(int wave_size, int heads, int* row_tile, int* head) {
  const int total = (int)gridDim.x, wave = (int)blockIdx.x / wave_size, place = (int)blockIdx.x - wave * wave_size;
  const int rank = wave & 1 ? total - 1 - ((wave >> 1) * wave_size + place) : ((wave + 1) >> 1) * wave_size + place;
  *row_tile = total / heads - 1 - rank / heads;
  *head = rank % heads;
}

// x and y as three pairs of bfloat16 whose sums are x and y to 24 bits (x in the low halves).  A value whose first
// part is not finite (infinite, NaN, or rounded up to infinity) has no further parts.
__device__ __forceinline__ void split3(float x, float y, uint32_t (&part)[3]) {
  constexpr float kLargest = 3.3895314e38f;
  part[0] = pack_pair(x, y);
  const float hx = low_bf16(part[0]), hy = high_bf16(part[0]);
  x = fabsf(hx) <= kLargest ? x - hx : 0.f;
  y = fabsf(hy) <= kLargest ? y - hy : 0.f;
  part[1] = pack_pair(x, y);
  part[2] = pack_pair(x - low_bf16(part[1]), y - high_bf16(part[1]));
}

}  // namespace einf
