// Products of float32 operands on the 5th-generation tensor cores, for recurrences by stretches (chunk_tcgen05.cu, delta_chunks.cu).
//
// Operands are float32 cut into three bfloat16 numbers each, rounded at every cut, so that a part is at most 2^-8 of the one before and the
// three hold all 24 bits.  Eight of the nine products of parts are made, as by mma_split (chunk_scan.cuh): what is left out is below 2^-32
// of a product.  (With six it is up to 2^-24.2, rms 2^-27.5: a product of two numbers no longer rounds to its float32 neighbour.)
// Operands lie in shared memory as [part][64 columns][rows of 128 bytes], 128-byte swizzle: such a tile is a K-major operand of its rows
// and an MN-major one of its columns.  The tensor cores cut off what a sum cannot hold instead of rounding it.  So every step of 16 of the
// two upper parts' product has an accumulator of its own, and registers add them up, rounding, while the seven small products of those
// steps (2^-7 of it at most) are made into one that they share: over eight steps 56 times a last place of theirs, 2^-24 of the whole at
// most and 2^-27 on average, is cut off, where a rounding after every step could cost eight times 2^-24.  With the upper product's steps
// in one accumulator too, outputs of constant decays (12 heads of 128 x 128, 2,048 tokens) were off by 2.0e-7 instead of 6.1e-8.
// The two products from six to eight cost 1.5 % of a delta rule layer (2,048 tokens, 24 heads: 269.0 us, so 273.2) and 0.8 % of one with
// constant decays (1,901 tokens, 12 heads of 128 x 128: 132.5, so 133.6).
#pragma once

#include "chunk_scan.cuh"
#include "ptx_sm100.cuh"

namespace ifx {

constexpr uint32_t kTcCut = 0x7f7f8000u;                   // from here on the upper part would round to infinity

__device__ __forceinline__ uint64_t tc_k_major(uint32_t addr) {         // rows of 128 bytes, groups of eight rows 1,024 apart
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t tc_mn_major(uint32_t addr, uint32_t next) {      // `next`: from 64 columns to the next
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((next >> 4) & 0x3FFF) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
constexpr uint32_t tc_idesc(int n, int a_mn, int b_mn) {                // M 128
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Two numbers, each the sum of its three parts, as pairs of bfloat16.
struct Cut {
  uint32_t part[3];
  __device__ __forceinline__ Cut(float x, float y) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
      part[p] = *reinterpret_cast<const uint32_t*>(&b);
      x -= __uint_as_float(part[p] << 16);
      y -= __uint_as_float(part[p] & 0xffff0000u);
    }
  }
};

// Four neighbouring numbers into a tile of ROWS rows and COLS columns.
template <int ROWS, int COLS>
__device__ __forceinline__ void tc_put(unsigned char* tile, int row, int c, float4 v) {
  const Cut a(v.x, v.y), b(v.z, v.w);
  unsigned char* at = tile + (c >> 6) * ROWS * 128 + row * 128 + ((((c >> 3) & 7) ^ (row & 7)) << 4) + (c & 4) * 2;
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(at + p * (COLS / 64) * ROWS * 128) = make_uint2(a.part[p], b.part[p]);
}
__device__ __forceinline__ uint32_t tc_largest(uint32_t m, float4 v) {
  return max(max(m, max(magnitude(v.x), magnitude(v.y))), max(magnitude(v.z), magnitude(v.w)));
}
// THREADS threads' reads of a tile: piece i of a thread is row i * (THREADS / (COLS / 4)) + thread / (COLS / 4), four columns.
template <int ROWS, int COLS, int THREADS>
struct TcTile {
  static constexpr int ACROSS = COLS / 4, PASS = THREADS / ACROSS, PIECES = ROWS / PASS;
  static constexpr uint32_t HALF = ROWS * 128, PART = (COLS / 64) * HALF, BYTES = 3 * PART;
  __device__ __forceinline__ static int row(int i) { return i * PASS + (int)threadIdx.x / ACROSS; }
  __device__ __forceinline__ static int col() { return ((int)threadIdx.x % ACROSS) * 4; }
};

// acc += x y^T over KSTEPS steps of 16 (x(part, step), y(part, step): operands).  Tensor memory from `at`: SLOTS accumulators of N columns, the
// first for the small products.  A thread adds up COLS columns of its lane from `col`, groups of 16 that lie SPREAD apart.  `meanwhile` runs under the first products.
// One warp issues, the upper products first: with the small ones by a second warp they delay the sums of the upper ones (139.6 us a layer
// of constant decays instead of 133.6).
// Two barriers, for the upper products of a round and for the end: one alone could complete twice before a thread looks.
// By all threads of the block, operands in place and in sight of the tensor cores; at the end nothing is at work any more as far as the
// others are concerned, and the issuer meets them at the next barrier.
template <int N, int KSTEPS, int SLOTS, int SPREAD = 16, int COLS, typename X, typename Y, typename Issue, typename Meanwhile>
__device__ __forceinline__ bool tc_product(float (&acc)[COLS], uint32_t at, uint32_t col, uint32_t bar, uint2& phase, bool issuer, X x, Y y, Issue issue,
                                           bool more, Meanwhile meanwhile) {
  constexpr int EACH = SLOTS - 1 < KSTEPS ? SLOTS - 1 : KSTEPS, ROUNDS = (KSTEPS + EACH - 1) / EACH;
  constexpr int SMALL = 7, PX[SMALL] = {1, 2, 2, 0, 1, 1, 0}, PY[SMALL] = {2, 1, 0, 2, 1, 0, 1};
  bool ok = true;
  // a round's accumulators among themselves first: one rounding of the whole sum a round
  auto column = [&](int c) { return col + (c / 16) * SPREAD + c % 16; };
  auto add = [&](uint32_t slot, int count) {
#pragma unroll
    for (int c = 0; c < COLS; c += 8) {
      float v[3][8];
#pragma unroll
      for (int j0 = 0; j0 < count; j0 += 2) {              // (two more at a time)
        tc_ld8(slot + j0 * N + column(c), v[1]);
        if (j0 + 1 < count) tc_ld8(slot + (j0 + 1) * N + column(c), v[2]);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float both = j0 + 1 < count ? v[1][i] + v[2][i] : v[1][i];
          v[0][i] = j0 == 0 ? both : v[0][i] + both;
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[c + i] += v[0][i];
    }
  };
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int k0 = r * EACH, k1 = k0 + EACH < KSTEPS ? k0 + EACH : KSTEPS;
    if (issuer) {
      tc_after();
      const uint32_t elected = elect_one();
#pragma unroll
      for (int ks = k0; ks < k1; ++ks) issue(at + (1 + ks - k0) * N, x(0, ks), y(0, ks), 0u, elected);
      umma_commit(bar, elected);
#pragma unroll
      for (int ks = k0; ks < k1; ++ks)
#pragma unroll
        for (int i = 0; i < SMALL; ++i) issue(at, x(PX[i], ks), y(PY[i], ks), more || ks > 0 || i > 0 ? 1u : 0u, elected);
      if (r == ROUNDS - 1) umma_commit(bar + 8, elected);
      __syncwarp();
    }
    if (r == 0) meanwhile();
    ok = __all_sync(0xffffffffu, mbar_wait(bar, phase.x & 1)) && ok;
    tc_after();
    add(at + N, k1 - k0);
    tc_before();
    ++phase.x;
    if (r < ROUNDS - 1) __syncthreads();                   // the accumulators are free again
  }
  ok = __all_sync(0xffffffffu, mbar_wait(bar + 8, phase.y & 1)) && ok;
  tc_after();
  ++phase.y;
  return ok;
}
// The small products, once, behind the last product of a sum.
template <int SPREAD = 16, int COLS>
__device__ __forceinline__ void tc_add_small(float (&acc)[COLS], uint32_t at, uint32_t col) {
#pragma unroll
  for (int c = 0; c < COLS; c += 8) {
    float v[8];
    tc_ld8(at + col + (c / 16) * SPREAD + c % 16, v);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[c + i] += v[i];
  }
  tc_before();
}

}  // namespace ifx
