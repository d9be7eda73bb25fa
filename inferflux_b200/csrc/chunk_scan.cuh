// Pieces that the scans over whole stretches of tokens share (chunk_scan.cu, delta_chunks.cu): products on the tensor
// cores of float32 operands, none of whose bits is lost, with float32 sums, and the layout of their shared memory.
#pragma once

#include "common.cuh"

namespace ifx {

constexpr int kChunk = 64;                 // tokens of a stretch
constexpr int kSub = 16;                   // tokens within which decays are multiplied up pair by pair
constexpr int kPitchV = 64 + 8;            // floats from a row of 64 to the next: the reads below meet every bank once
constexpr int kPitchA = 64 + 4;

// What `splits` refuses, infinities and what is not a number, would come out of a product as something else than of a scan.
// Whoever makes a number that is to be split looks at it first, and a stretch that holds another one goes token by token.
constexpr uint32_t kSplitLimit = 0x7f800000u;
__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }
__device__ __forceinline__ bool splits(float x) { return magnitude(x) < kSplitLimit; }
__device__ __forceinline__ bool splits(float4 v) { return splits(v.x) && splits(v.y) && splits(v.z) && splits(v.w); }
// Two float32, each as the sum of three bfloat16 of 8 bits: the upper half of its bits, the upper half of what that leaves, the
// rest.  All 24 bits are kept.
struct Split {
  uint32_t hi, mid, lo;
  __device__ __forceinline__ void set(float x, float y) {
    hi = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
    y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
    mid = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
    y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
    lo = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
  }
};
__device__ __forceinline__ void mma_pairs(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
struct FragA { Split v[4]; };              // 16 rows x 16 of the inner size
struct FragB { Split v[2]; };              // 8 columns x 16 of the inner size
// c += a b.  The product of the two smallest parts (below 2^-29 of the whole) is left out.  The tensor cores cut off what a sum cannot
// hold instead of rounding it, so a sum that stays in their accumulator over many steps drifts to zero.  Here a step of 16 is summed
// there alone: the products of the upper parts have 16 bits each, and their sum loses next to nothing; what is cut off the sum of the
// others is below 2^-27 of the whole.  Both meet, and join the steps before, by additions that round.
__device__ __forceinline__ void mma_split(float (&c)[4], const FragA& a, const FragB& b) {
  float t[4] = {0.0f, 0.0f, 0.0f, 0.0f}, r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#define IFX_PAIR(to, x, y) mma_pairs(to, a.v[0].x, a.v[1].x, a.v[2].x, a.v[3].x, b.v[0].y, b.v[1].y)
  IFX_PAIR(t, hi, hi);
  IFX_PAIR(r, lo, mid);
  IFX_PAIR(r, mid, lo);
  IFX_PAIR(r, lo, hi);
  IFX_PAIR(r, hi, lo);
  IFX_PAIR(r, mid, mid);
  IFX_PAIR(r, mid, hi);
  IFX_PAIR(r, hi, mid);
#undef IFX_PAIR
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += t[i] + r[i];
}
// A product of many factors as the sum of two numbers, the second one what the first one's roundings left out: the same decay
// multiplied up over 64 tokens would otherwise carry the same error from stretch to stretch.
struct Product {
  float hi = 1.0f, lo = 0.0f;
  __device__ __forceinline__ void times(float w) {
    const float p = hi * w;
    lo = fmaf(lo, w, fmaf(hi, w, -p));
    hi = p;
  }
  __device__ __forceinline__ float value() const { return hi + lo; }
};
// Operands whose inner size runs along a row of shared memory.  A lane takes two neighbouring numbers of either eight, 2 t and
// 2 t + 1 for t = lane % 4, in one read; both operands of a product do, so the order within a step of 16 is the same for both.
// Row pitch 8 modulo 32 floats.
__device__ __forceinline__ void load_a_rows(FragA& f, const float* p, int pitch, int lane) {
  const float* at = p + (lane >> 2) * pitch + 2 * (lane & 3);
  const float2 x = *reinterpret_cast<const float2*>(at), x8 = *reinterpret_cast<const float2*>(at + 8);
  const float2 y = *reinterpret_cast<const float2*>(at + 8 * pitch), y8 = *reinterpret_cast<const float2*>(at + 8 * pitch + 8);
  f.v[0].set(x.x, x8.x);
  f.v[1].set(y.x, y8.x);
  f.v[2].set(x.y, x8.y);
  f.v[3].set(y.y, y8.y);
}
__device__ __forceinline__ float2 read_b_rows(const float* p, int pitch, int lane) {
  return *reinterpret_cast<const float2*>(p + (lane >> 2) * pitch + 2 * (lane & 3));
}
__device__ __forceinline__ void load_b_rows(FragB& f, const float* p, int pitch, int lane) {
  const float2 x = read_b_rows(p, pitch, lane), x8 = read_b_rows(p + 8, pitch, lane);
  f.v[0].set(x.x, x8.x);
  f.v[1].set(x.y, x8.y);
}
// The same of rows that are not paired up, for a product whose other operand has its inner size across rows.  Row pitch 4
// modulo 32 floats.
__device__ __forceinline__ void load_a_single(FragA& f, const float* p, int pitch, int lane) {
  const float* at = p + (lane >> 2) * pitch + (lane & 3);
  f.v[0].set(at[0], at[8]);
  f.v[1].set(at[8 * pitch], at[8 * pitch + 8]);
  f.v[2].set(at[4], at[12]);
  f.v[3].set(at[8 * pitch + 4], at[8 * pitch + 12]);
}
// Operands whose inner size runs across rows.  Row pitch 8 modulo 32 floats.
__device__ __forceinline__ void load_a_columns(FragA& f, const float* p, int pitch, int lane) {
  const float* at = p + (lane & 3) * pitch + (lane >> 2);
  f.v[0].set(at[0], at[8 * pitch]);
  f.v[1].set(at[8], at[8 * pitch + 8]);
  f.v[2].set(at[4 * pitch], at[12 * pitch]);
  f.v[3].set(at[4 * pitch + 8], at[12 * pitch + 8]);
}
__device__ __forceinline__ void load_b_columns(FragB& f, const float* p, int pitch, int lane) {
  const float* at = p + (lane & 3) * pitch + (lane >> 2);
  f.v[0].set(at[0], at[8 * pitch]);
  f.v[1].set(at[4 * pitch], at[12 * pitch]);
}

// Stretch `index` of the step's spans of min_span tokens and more: its request, first flat token and tokens.  Stretches of a
// request lie side by side.
// (`per`: tokens of a stretch)
__device__ __forceinline__ int chunks_of(int span, int min_span, int per = kChunk) { return span < min_span ? 0 : (span + per - 1) / per; }
__device__ __forceinline__ bool chunk_of(const int* __restrict__ cu_seqlens, int requests, int min_span, int index, int& first, int& n,
                                         int per = kChunk) {
  int before = 0;
  for (int r = 0; r < requests; ++r) {
    const int lo = cu_seqlens[r], span = cu_seqlens[r + 1] - lo, chunks = chunks_of(span, min_span, per);
    if (index < before + chunks) {
      first = lo + (index - before) * per;
      n = min(per, span - (index - before) * per);
      return true;
    }
    before += chunks;
  }
  return false;
}
__device__ __forceinline__ int chunks_before(const int* __restrict__ cu_seqlens, int min_span, int request, int per = kChunk) {
  int before = 0;
  for (int r = 0; r < request; ++r) before += chunks_of(cu_seqlens[r + 1] - cu_seqlens[r], min_span, per);
  return before;
}
// The most stretches that num_tokens of num_requests can make.
inline int chunks_at_most(int num_tokens, int num_requests, int min_span, int per = kChunk) {
  const int spans = num_tokens / (min_span > 1 ? min_span : 1);
  return num_tokens / per + (spans < num_requests ? spans : num_requests);
}

enum { CHUNK_CHANNEL = 0, CHUNK_STEP = 1, CHUNK_CONSTANT = 2, CHUNK_WKV = 3 };

struct ChunkArgs {
  const float* q; long long q_stride;
  const float* k; long long k_stride;
  const float* v; long long v_stride;
  const float* raw; long long raw_stride;
  float* state; long long state_slot_stride;
  const int* req_slot; const int* cu_seqlens;
  float* out;                                   // [T, heads dv]
  const float* step_bias; const float* log_rate; const float* skip; const float* rate;      // per head
  const float* w0; const float* u;              // CHUNK_WKV: per head and key channel
  int requests, min_span, heads, groups, dv;    // shorter spans are left to the scans token by token
  float inv_tau, q_scale;
  float* local;                                 // [stretches, heads, dv, dk]: what a stretch adds, then the state in front of it
  float* total;                                 // decays of a whole stretch: [stretches, heads, dk], or [stretches, heads] as two numbers each
  float* reach;                                 // queries times decays since the stretch's beginning [T, heads dk], or decays [T, heads]
  int key_rows;                                 // the request's state is [head, key channel, value channel]
  const float* x; float* prev_state; int C;     // CHUNK_WKV: the step's input rows, where the last one of a request goes
};

__device__ __forceinline__ float chunk_log_sigmoid(float x) { return fminf(x, 0.0f) - log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float chunk_softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

}  // namespace ifx
