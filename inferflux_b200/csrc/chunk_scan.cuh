// Pieces that the scans over whole stretches of tokens share (chunk_scan.cu, delta_chunks.cu): products on the tensor
// cores whose result is as exact as a float32 multiply-add chain, and the layout of their shared memory.
#pragma once

#include "common.cuh"

namespace ifx {

constexpr int kChunk = 64;                 // tokens of a stretch
constexpr int kSub = 16;                   // tokens within which decays are multiplied up pair by pair
constexpr int kPitchV = 64 + 8;            // floats from a row of 64 to the next: the reads below meet every bank once
constexpr int kPitchA = 64 + 4;

// A float32 as the sum of two numbers of 11 bits each, both rounded to the nearest: what is left out is below 2^-22 of it.  By
// integer additions on the bits, since conversions run at a fraction of their rate; the product does not look at the 13 lowest
// bits of an operand, so the small part's stay where they are.  Finite numbers only: a NaN would be lost.
struct Split {
  uint32_t hi, lo;
  __device__ __forceinline__ void set(float x) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi)) + 0x1000u;
  }
};
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
struct FragA { Split v[4]; };              // 16 rows x 8 of the inner size
struct FragB { Split v[2]; };              // 8 columns x 8 of the inner size
// c += a b with both operands split; the product of the two small parts (below 2^-22 of the whole) is left out.
__device__ __forceinline__ void mma_split(float (&c)[4], const FragA& a, const FragB& b) {
  mma_tf32(c, a.v[0].lo, a.v[1].lo, a.v[2].lo, a.v[3].lo, b.v[0].hi, b.v[1].hi);
  mma_tf32(c, a.v[0].hi, a.v[1].hi, a.v[2].hi, a.v[3].hi, b.v[0].lo, b.v[1].lo);
  mma_tf32(c, a.v[0].hi, a.v[1].hi, a.v[2].hi, a.v[3].hi, b.v[0].hi, b.v[1].hi);
}
// Operands whose inner size runs along a row of shared memory.  A lane takes two neighbouring numbers of it, 2 t and 2 t + 1 for
// t = lane % 4, in one read; both operands of a product do, so the order within a step of eight is the same for both.
// Row pitch 8 modulo 32 floats.
__device__ __forceinline__ void load_a_rows(FragA& f, const float* p, int pitch, int lane) {
  const float2 x = *reinterpret_cast<const float2*>(p + (lane >> 2) * pitch + 2 * (lane & 3));
  const float2 y = *reinterpret_cast<const float2*>(p + ((lane >> 2) + 8) * pitch + 2 * (lane & 3));
  f.v[0].set(x.x);
  f.v[1].set(y.x);
  f.v[2].set(x.y);
  f.v[3].set(y.y);
}
__device__ __forceinline__ float2 read_b_rows(const float* p, int pitch, int lane) {
  return *reinterpret_cast<const float2*>(p + (lane >> 2) * pitch + 2 * (lane & 3));
}
__device__ __forceinline__ void load_b_rows(FragB& f, const float* p, int pitch, int lane) {
  const float2 x = read_b_rows(p, pitch, lane);
  f.v[0].set(x.x);
  f.v[1].set(x.y);
}
// The same of rows that are not paired up, for a product whose other operand has its inner size across rows.  Row pitch 4
// modulo 32 floats.
__device__ __forceinline__ void load_a_single(FragA& f, const float* p, int pitch, int lane) {
  const float* at = p + (lane >> 2) * pitch + (lane & 3);
  f.v[0].set(at[0]);
  f.v[1].set(at[8 * pitch]);
  f.v[2].set(at[4]);
  f.v[3].set(at[8 * pitch + 4]);
}
// Operands whose inner size runs across rows.  Row pitch 8 modulo 32 floats.
__device__ __forceinline__ void load_a_columns(FragA& f, const float* p, int pitch, int lane) {
  const float* at = p + (lane & 3) * pitch + (lane >> 2);
  f.v[0].set(at[0]);
  f.v[1].set(at[8]);
  f.v[2].set(at[4 * pitch]);
  f.v[3].set(at[4 * pitch + 8]);
}
__device__ __forceinline__ void load_b_columns(FragB& f, const float* p, int pitch, int lane) {
  const float* at = p + (lane & 3) * pitch + (lane >> 2);
  f.v[0].set(at[0]);
  f.v[1].set(at[4 * pitch]);
}

// Stretch `index` of the step: its request, first flat token and tokens.  Stretches of a request lie side by side.
__device__ __forceinline__ bool chunk_of(const int* __restrict__ cu_seqlens, int requests, int index, int& first, int& n) {
  int before = 0;
  for (int r = 0; r < requests; ++r) {
    const int lo = cu_seqlens[r], span = cu_seqlens[r + 1] - lo, chunks = (span + kChunk - 1) / kChunk;
    if (index < before + chunks) {
      first = lo + (index - before) * kChunk;
      n = min(kChunk, span - (index - before) * kChunk);
      return true;
    }
    before += chunks;
  }
  return false;
}
__device__ __forceinline__ int chunks_before(const int* __restrict__ cu_seqlens, int request) {
  int before = 0;
  for (int r = 0; r < request; ++r) before += (cu_seqlens[r + 1] - cu_seqlens[r] + kChunk - 1) / kChunk;
  return before;
}
// The most stretches that num_tokens of num_requests can make.
inline int chunks_at_most(int num_tokens, int num_requests) { return num_tokens / kChunk + num_requests; }

__device__ __forceinline__ bool all_finite(float4 v) { return isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w); }

}  // namespace ifx
