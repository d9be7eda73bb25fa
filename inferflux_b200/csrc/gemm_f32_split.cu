// Float32 matrix product C[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) on the 5th-generation tensor cores, at 32-bit precision.
//
// Every operand is cut into three bfloat16 numbers that add up to it exactly: the number rounded to 8 bits, what is left rounded to 8
// bits, and what is left then (7 bits at most).  An output is the sum of six products of parts: hi hi; mid hi, hi mid, mid mid, lo hi,
// hi lo.  What is left out (mid lo, lo mid, lo lo) is below 2^-23.9 of a product's size, of either sign.  The tensor cores cut off
// when they add.  So products hi hi, which have 16 bits, get an accumulator of their own, and a fresh one every 64 k, whose sums are
// added up in registers with rounded float32 additions, k ascending; the other five, 2^-8 of them, run in a second accumulator that is
// added every 16 chunks.
// Errors against 64 bits (2-norm, normal numbers; chain of multiply-adds and this): K 1,288 6.5e-7 and 1.0e-7; 8,960 17e-7 and 1.2e-7
// (2.3e-7 where K is not in slices); 18,944 25e-7 and 1.7e-7.  Rows with one, two, four, eight numbers that are not 0: 2.5e-8 and
// 2.6e-8; 3.0 and 3.0 to 4.1; 4.0 and 3.4 to 4.9; 5.3 and 4.0 to 5.9: the slices and the second accumulator round once more.  (Parts
// cut off instead of rounded, all six products in one accumulator: 1.0e-7 in these four, 4.6e-7 at most; dense rows 1.4e-7 to 2.5e-7.)
//
// An output's additions depend on K and N alone (how K is cut into slices does), never on the number of rows, so a row's bits
// are the same whatever other rows share the launch.  Parts of a number below 2^-109 end at bfloat16's smallest, 2^-133.  That is
// nothing in a result of 2^-60 or more whose operands are below 2^35.  All other results are made again as the plain chain of
// multiply-adds, a tile at a time by the block that made them: those below 2^-60, those that are not finite, and those of a row (of
// either operand) with a number of 2^35 or more, which puts a NaN into its row's first part.  So infinities, NaN and overflow behave
// as there.
//
// Swapped operands: 128 weight rows are the lanes of tensor memory, up to 128 token rows the columns.  Persistent blocks:
//
//   warp 0        TMA: weights as they are (float32, [128 x 64] a chunk), the tokens' three planes (split_rows_kernel) as bfloat16
//   warps 2-9     cut a chunk's weight rows, read from shared memory, and store the three parts into tensor memory (the products'
//                 A operand); four warps the even chunks, four the odd ones (one group of four: 121 us instead of 109)
//   warp 1        24 tcgen05.mma a chunk (M 128, N tokens, K 16, A from tensor memory), hi hi first: its accumulator is read while
//                 others run
//   warps 10-17   add finished accumulators to their registers, half the columns each four; behind the last chunk store,
//                 neighbouring lanes neighbouring columns of a row
//
// Bound: the tensor pipe for many rows (1,000 rows of 3,584 -> 37,888: 1,148 us, six products at 1.42 PFLOP/s); cutting and
// reading the weights for few.  Measured, gemm_f32_tiles_kernel -> this with both kernels beside it (us): 333 rows, 1,536 ->
// 17,920: 485 -> 95; 8,960 -> 1,536: 310 -> 71; one row: 33 -> 30 and 107 -> 23; 150 rows, 18,944 -> 3,584: 650 -> 141.  Of 333 rows
// one that is not finite: 232 and 357; all of them: 1,259 and 534.  Weights that are all zero: 3 times the time of others.
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace ifx {

constexpr int kSplitRows = 128, kSplitK = 64;                    // weight rows of a tile, k of a chunk
constexpr uint32_t kSplitWBytes = kSplitRows * kSplitK * 4;      // a chunk of float32 weights
constexpr int kSplitMaxStages = 4, kSplitTStages = 3;            // of the weights' ring at most, of the tokens'
constexpr int kSplitThreads = 576;
constexpr int kSplitPartCols = kSplitK / 2;                      // tensor memory columns of one part of a chunk
constexpr int kSplitACols = 3 * kSplitPartCols;
constexpr int kSplitBig = 96;                                    // columns of the first of two accumulators
constexpr int kSplitDrain = 16;                                  // chunks of the five smaller products between two additions

// a, b -> three pairs of bfloat16 (a below, b above); `largest` of the magnitudes so far (NaN do not count).
__device__ __forceinline__ void cut_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo, float& largest) {
  auto rounded = [](float x, float y) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&v);
  };
  auto below = [](uint32_t pair) { return __uint_as_float(pair << 16); };
  auto above = [](uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); };
  hi = rounded(a, b);
  const float ra = a - below(hi), rb = b - above(hi);
  mid = rounded(ra, rb);
  lo = __byte_perm(__float_as_uint(ra - below(mid)), __float_as_uint(rb - above(mid)), 0x7632);
  asm("{\n\t.reg .f32 x, y;\n\tabs.f32 x, %1;\n\tabs.f32 y, %2;\n\tmax.f32 %0, %0, x, y;\n\t}" : "+f"(largest) : "f"(a), "f"(b));
}
constexpr uint32_t kNanPair = 0x7fff7fffu;
constexpr float kSplitLargest = 34359738368.0f;                  // 2^35: from here on a row is made again
constexpr float kSplitSmallest = 8.673617379884035e-19f;         // 2^-60: results below are

// planes [3, rows, K] bfloat16 <- x [rows, K] float32, eight numbers a thread.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ planes, long long n8) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= n8) return;
  const float4 a = reinterpret_cast<const float4*>(x)[2 * i], b = reinterpret_cast<const float4*>(x)[2 * i + 1];
  uint4 hi, mid, lo;
  float largest = 0.0f;
  cut_pair(a.x, a.y, hi.x, mid.x, lo.x, largest);
  cut_pair(a.z, a.w, hi.y, mid.y, lo.y, largest);
  cut_pair(b.x, b.y, hi.z, mid.z, lo.z, largest);
  cut_pair(b.z, b.w, hi.w, mid.w, lo.w, largest);
  if (!(largest < kSplitLargest)) hi.x = kNanPair;
  uint4* out = reinterpret_cast<uint4*>(planes);
  out[i] = hi;
  out[n8 + i] = mid;
  out[2 * n8 + i] = lo;
}

// Whether a result has to be made again (see the top), and what stands in its place until then.
__device__ __forceinline__ bool made_again(float v) { return !(fabsf(v) < INFINITY) || fabsf(v) < kSplitSmallest; }
constexpr uint32_t kWasZero = 0x7fc00001u, kWasOther = 0x7fffffffu;              // NaN both
__device__ __forceinline__ float placeholder(float v) { return __uint_as_float(v == 0.0f ? kWasZero : kWasOther); }

// Results [m0 .. m0 + 32) x [n0 .. n0 + COLS) that are NaN, made again as the chain of multiply-adds (k ascending, then the bias).
// All threads of a block fetch, four warps multiply: 8 rows and every 32nd column a thread.  smem: again_floats(COLS), free.  Zeros of
// rows that hold nothing else are not multiplied out: they are the results that come here in earnest.
constexpr int kAgainRows = 32, kAgainK = 32, kAgainPitch = kAgainK + 4, kAgainStages = 3;
constexpr int again_floats(int cols) { return (kAgainRows + cols) * (kAgainStages * kAgainPitch + 1); }
template <int COLS, int THREADS>
__device__ __noinline__ void make_again(float* smem, const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                                        float* out, int M, int N, int K, int m0, int n0) {
  constexpr int LINES = kAgainRows + COLS, EACH = COLS / 32;                     // lines: rows of A, then rows of W
  static_assert(EACH <= 4 && THREADS >= 128, "");
  const int tid = threadIdx.x, lane = tid & 31, row = (tid >> 5) * 8;
  uint32_t* line_s = reinterpret_cast<uint32_t*>(smem + LINES * kAgainStages * kAgainPitch);          // the largest magnitude of a line
  auto place = [&](int r, int j) { return out + (size_t)(m0 + row + r) * N + n0 + j * 32 + lane; };
  unsigned need = 0, zeros = 0;                                                  // bit 8 j + r
  if (tid < 128) {
#pragma unroll
    for (int j = 0; j < EACH; ++j)
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (m0 + row + r < M && n0 + j * 32 + lane < N) {
          const float v = *place(r, j);
          if (isnan(v)) need |= 1u << (8 * j + r);
          if (__float_as_uint(v) == kWasZero) zeros |= 1u << (8 * j + r);
        }
  }
  if (!__syncthreads_or(need != 0)) return;
  auto line = [&](int i) {
    return i < kAgainRows ? A + (size_t)min(m0 + i, M - 1) * K : W + (size_t)min(n0 + i - kAgainRows, N - 1) * K;
  };
  const unsigned all = need;
  if (__syncthreads_or(zeros != 0)) {                                            // of these, the ones of a line of zeros stay
    for (int e = tid; e < LINES; e += THREADS) line_s[e] = 0;
    __syncthreads();
    for (int e = tid; e < LINES * 16; e += THREADS) {
      const float* src = line(e >> 4);
      uint32_t most = 0;
#pragma unroll 4
      for (int k = (e & 15) * 4; k < K; k += 64) {
        const uint4 v = *reinterpret_cast<const uint4*>(src + k);
        most = max(max(most, max(v.x & 0x7fffffffu, v.y & 0x7fffffffu)), max(v.z & 0x7fffffffu, v.w & 0x7fffffffu));
      }
      atomicMax(&line_s[e >> 4], most);
    }
    __syncthreads();
    if (zeros) {
#pragma unroll
      for (int i = 0; i < 8 * EACH; ++i)
        if ((zeros >> i & 1u) && (line_s[row + i % 8] == 0 || line_s[kAgainRows + i / 8 * 32 + lane] == 0)) need &= ~(1u << i);
    }
  }
  float acc[EACH][8] = {};
  if (__syncthreads_or(need != 0)) {
    unsigned rows = __reduce_or_sync(0xffffffffu, need);
    rows = (rows | rows >> 8 | rows >> 16 | rows >> 24) & 0xffu;
    auto fetch = [&](int k0) {
      float* to = smem + k0 / kAgainK % kAgainStages * LINES * kAgainPitch;
      for (int e = tid; e < LINES * (kAgainK / 4); e += THREADS) {
        const int i = e / (kAgainK / 4), k = e % (kAgainK / 4) * 4;
        if (k0 + k < K)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(to + i * kAgainPitch + k)), "l"(line(i) + k0 + k) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int k0 = 0; k0 < (kAgainStages - 1) * kAgainK; k0 += kAgainK) fetch(k0);
    for (int k0 = 0; k0 < K; k0 += kAgainK) {
      fetch(k0 + (kAgainStages - 1) * kAgainK);
      asm volatile("cp.async.wait_group %0;" ::"n"(kAgainStages - 1) : "memory");
      __syncthreads();
      const float* from = smem + k0 / kAgainK % kAgainStages * LINES * kAgainPitch;
      const int left = min(kAgainK, K - k0);
      auto step = [&](int k, unsigned which) {
        float4 w[EACH];
#pragma unroll
        for (int j = 0; j < EACH; ++j) w[j] = *reinterpret_cast<const float4*>(from + (kAgainRows + j * 32 + lane) * kAgainPitch + k);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          if (which >> r & 1u) {
            const float4 x = *reinterpret_cast<const float4*>(from + (row + r) * kAgainPitch + k);
#pragma unroll
            for (int j = 0; j < EACH; ++j)
              acc[j][r] = fmaf(x.w, w[j].w, fmaf(x.z, w[j].z, fmaf(x.y, w[j].y, fmaf(x.x, w[j].x, acc[j][r]))));
          }
        }
      };
      if (rows & (rows - 1)) {                                     // more than one row: all eight
#pragma unroll 1
        for (int k = 0; k < left; k += 4) step(k, 0xffu);
      } else if (rows) {
#pragma unroll 1
        for (int k = 0; k < left; k += 4) step(k, rows);
      }
      __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
#pragma unroll
  for (int j = 0; j < EACH; ++j)
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (all >> (8 * j + r) & 1u) {
        const float v = need >> (8 * j + r) & 1u ? acc[j][r] : 0.0f;
        *place(r, j) = bias ? v + bias[n0 + j * 32 + lane] : v;
      }
  __syncthreads();
}

__device__ __forceinline__ void split_tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void split_tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ uint64_t split_smem_desc(uint32_t addr) {
  // K-major tile of 128-byte rows, 128-byte swizzle: 8-row groups 1024 bytes apart.
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void split_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

struct SplitArgs {
  const float *A, *W, *bias;
  float* out;                          // [M, N], or [slices, M, N] where slices > 1
  int M, N, K, m_tiles, n_tiles, slices, slice_chunks, chunks, nt, w_log;     // w_log: log2 of the weights' stages
  int* error_flag;
};

// NT: registers for sums (token rows of a tile at most); args.nt of them are there.
template <int NT>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_t, const SplitArgs args) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bars[4 * kSplitMaxStages + 10];
  __shared__ uint32_t tmem_holder;
  __shared__ int again_s;                                          // a result of this block has to be made again
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int nt = args.nt, w_log = args.w_log, w_stages = 1 << w_log;
  constexpr int t_stages = kSplitTStages;
  const uint32_t plane_bytes = (uint32_t)nt * kSplitK * 2, t_bytes = 3 * plane_bytes;
  const uint32_t w_smem = smem_addr(smem), t_smem = w_smem + w_stages * kSplitWBytes;
  const uint32_t w_full = smem_addr(bars), w_empty = w_full + 8 * kSplitMaxStages, t_full = w_empty + 8 * kSplitMaxStages,
                 t_empty = t_full + 8 * kSplitMaxStages, a_full = t_empty + 8 * kSplitMaxStages, a_empty = a_full + 16, big_full = a_empty + 16, big_empty = big_full + 16,
                 small_full = big_empty + 16, small_empty = small_full + 8;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int tiles = args.m_tiles * args.n_tiles * args.slices;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSplitMaxStages; ++s) {
      mbar_init(w_full + 8 * s, 1);
      mbar_init(w_empty + 8 * s, 4);
      mbar_init(t_full + 8 * s, 1);
      mbar_init(t_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(a_full + 8 * b, 4);
      mbar_init(a_empty + 8 * b, 1);
      mbar_init(big_full + 8 * b, 1);
      mbar_init(big_empty + 8 * b, 8);
    }
    mbar_init(small_full, 1);
    mbar_init(small_empty, 8);
    again_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_holder;
  // Tensor memory: hi hi, twice where three accumulators of a tile fit (few tokens, whose products do not last until the first has
  // been read: one row, 3,584 -> 37,888, 104 -> 97 us), the rest of the products, the parts twice.
  const int bigs = nt <= kSplitBig ? 2 : 1;
  const uint32_t small = tmem + (bigs == 2 ? 2 * kSplitBig : kSplitRows), a_tmem = tmem + 512 - 2 * kSplitACols;

  // A tile: token tiles fastest, so that blocks running at a time read the same weights; then slices of K, then weight rows.
  auto slice_of = [&](int t, int& m_tile, int& n_tile, int& slice, int& c0, int& c1) {
    m_tile = t % args.m_tiles;
    const int r = t / args.m_tiles;
    slice = r % args.slices;
    n_tile = r / args.slices;
    c0 = slice * args.slice_chunks;
    c1 = min(args.chunks, c0 + args.slice_chunks);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    if (lane == 0) {
      int i = 0;                                                   // chunks so far
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        int mt, ntile, slice, c0, c1;
        slice_of(t, mt, ntile, slice, c0, c1);
        for (int c = c0; c < c1; ++c, ++i) {
          const int ws = i & (w_stages - 1), ts = i % t_stages;
          if (i >= w_stages) ok = mbar_wait(w_empty + 8 * ws, ((i >> w_log) & 1) ^ 1);
          if (!ok) break;
          mbar_expect_tx(w_full + 8 * ws, kSplitWBytes);
          const uint32_t dst = w_smem + ws * kSplitWBytes;
          tma_load_2d(dst, &map_w, c * kSplitK, ntile * kSplitRows, w_full + 8 * ws);
          tma_load_2d(dst + kSplitWBytes / 2, &map_w, c * kSplitK + 32, ntile * kSplitRows, w_full + 8 * ws);
          if (i >= t_stages) ok = mbar_wait(t_empty + 8 * ts, ((i / t_stages) & 1) ^ 1);
          if (!ok) {
            mbar_wait(w_full + 8 * ws, (i >> w_log) & 1);        // not counted below: it has no tokens
            break;
          }
          mbar_expect_tx(t_full + 8 * ts, t_bytes);
          for (int p = 0; p < 3; ++p)
            tma_load_2d(t_smem + ts * t_bytes + p * plane_bytes, &map_t, c * kSplitK, p * args.M + mt * nt, t_full + 8 * ts);
        }
      }
      if (!ok) {
        atomicExch(args.error_flag, 61);
        for (int j = max(0, i - w_stages); j < i; ++j) mbar_wait(w_full + 8 * (j & (w_stages - 1)), (j >> w_log) & 1);
        for (int j = max(0, i - t_stages); j < i; ++j) mbar_wait(t_full + 8 * (j % t_stages), (j / t_stages) & 1);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ products
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(kSplitRows >> 4) << 24);
    const uint32_t elected = elect_one();
    const uint64_t plane_step = plane_bytes >> 4;
    int i = 0, sums = 0;                                           // chunks, uses of the second accumulator so far
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int mt, ntile, slice, c0, c1;
      slice_of(t, mt, ntile, slice, c0, c1);
      for (int c = c0; c < c1; ++c, ++i) {
        const int buf = i & 1, ts = i % t_stages;
        const bool fresh = (c - c0) % kSplitDrain == 0;
        ok = mbar_wait(t_full + 8 * ts, (i / t_stages) & 1) && mbar_wait(a_full + 8 * buf, (i >> 1) & 1);
        const int big = i & (bigs - 1), use = i >> (bigs - 1);
        if (ok && use > 0) ok = mbar_wait(big_empty + 8 * big, (use & 1) ^ 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = a_tmem + buf * kSplitACols;
        const uint64_t b = split_smem_desc(t_smem + ts * t_bytes);
#pragma unroll
        for (int k = 0; k < kSplitK / 16; ++k) umma_ts(tmem + big * kSplitBig, a + k * 8, b + 2 * k, idesc, k > 0 ? 1u : 0u, elected);
        umma_commit(big_full + 8 * big, elected);
        if (fresh && sums > 0) ok = mbar_wait(small_empty, (sums & 1) ^ 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // (part of the weights, part of the tokens): 0 hi, 1 mid, 2 lo; the smallest products first
        constexpr int WP[5] = {2, 0, 1, 1, 0}, TP[5] = {0, 2, 1, 0, 1};
#pragma unroll
        for (int p = 0; p < 5; ++p)
#pragma unroll
          for (int k = 0; k < kSplitK / 16; ++k)
            umma_ts(small, a + WP[p] * kSplitPartCols + k * 8, b + TP[p] * plane_step + 2 * k, idesc, (!fresh || p > 0 || k > 0) ? 1u : 0u, elected);
        umma_commit(t_empty + 8 * ts, elected);
        umma_commit(a_empty + 8 * buf, elected);
        if (c + 1 == c1 || (c + 1 - c0) % kSplitDrain == 0) {
          umma_commit(small_full, elected);
          ++sums;
        }
      }
    }
    if (!ok && lane == 0) atomicExch(args.error_flag, 62);
    __syncwarp();
  } else if (warp < 10) {
    // ------------------------------------------------------------------ a weight row each: cut into parts
    const int row = (warp & 3) * 32 + lane, group = (warp - 2) >> 2;
    int i = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int mt, ntile, slice, c0, c1;
      slice_of(t, mt, ntile, slice, c0, c1);
      for (int c = c0; c < c1; ++c, ++i) {
        const int buf = i & 1, ws = i & (w_stages - 1);
        if (buf != group) continue;
        ok = mbar_wait(w_full + 8 * ws, (i >> w_log) & 1);
        if (ok && i >= 2) ok = mbar_wait(a_empty + 8 * buf, ((i >> 1) & 1) ^ 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t base = a_tmem + ((uint32_t)((warp & 3) * 32) << 16) + buf * kSplitACols;
#pragma unroll
        for (int h = 0; h < 2; ++h) {                              // 32 k: a row of 128 bytes, 16-byte pieces swizzled
          const unsigned char* src = smem + (size_t)ws * kSplitWBytes + h * (kSplitWBytes / 2) + row * 128;
          uint32_t hi[16], mid[16], lo[16];
          float largest = 0.0f;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 v = *reinterpret_cast<const float4*>(src + ((q ^ (row & 7)) << 4));
            cut_pair(v.x, v.y, hi[2 * q], mid[2 * q], lo[2 * q], largest);
            cut_pair(v.z, v.w, hi[2 * q + 1], mid[2 * q + 1], lo[2 * q + 1], largest);
          }
          if (!(largest < kSplitLargest)) hi[0] = kNanPair;
          split_tmem_st16(base + h * 16, hi);
          split_tmem_st16(base + kSplitPartCols + h * 16, mid);
          split_tmem_st16(base + 2 * kSplitPartCols + h * 16, lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        fence_proxy_async_smem();                                  // the reads above before the next TMA write
        __syncwarp();
        if (lane == 0) {
          split_arrive(a_full + 8 * buf);
          split_arrive(w_empty + 8 * ws);
        }
      }
    }
    if (!ok && lane == 0) atomicExch(args.error_flag, 63);
  } else {
    // ------------------------------------------------------------------ sums of chunks, results
    constexpr int COLS = NT / 2;
    const int quarter = warp & 3, first = (warp - 10) / 4 * COLS;    // token columns first .. first + COLS
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    int i = 0, sums = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int mt, ntile, slice, c0, c1;
      slice_of(t, mt, ntile, slice, c0, c1);
      float sum[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) sum[j] = 0.0f;
      auto add = [&](uint32_t acc, uint32_t full, uint32_t empty, int use) {
        if (!mbar_wait(full, use & 1)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int j0 = 0; j0 < COLS; j0 += 16) {
          if (first + j0 < nt) {
            uint32_t r[16];
            split_tmem_ld16(acc + lanes + first + j0, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j0 + j] += __uint_as_float(r[j]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) split_arrive(empty);
        return true;
      };
      for (int c = c0; c < c1 && ok; ++c, ++i) {
        const int big = i & (bigs - 1);
        ok = add(tmem + big * kSplitBig, big_full + 8 * big, big_empty + 8 * big, i >> (bigs - 1));
        if (ok && (c + 1 == c1 || (c + 1 - c0) % kSplitDrain == 0)) ok = add(small, small_full, small_empty, sums++);
      }
      if (!ok) break;
      const int n = ntile * kSplitRows + quarter * 32 + lane, m0 = mt * nt + first;
      const int cols = min(min(COLS, nt - first), args.M - m0);
      if (n < args.N) {
        float* out = args.out + (size_t)slice * args.M * args.N + n;
        const bool whole = args.slices == 1;
        const float b = whole && args.bias ? args.bias[n] : 0.0f;
        bool again = false;
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
          if (j < cols) {
            const bool lost = whole && made_again(sum[j]);
            again = again || lost;
            out[(size_t)(m0 + j) * args.N] = lost ? placeholder(sum[j]) : sum[j] + b;
          }
        }
        if (again) again_s = 1;
      }
    }
    if (!ok && lane == 0) atomicExch(args.error_flag, 64);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (again_s == 0) return;                                        // (set in front of the barrier above)
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    int mt, ntile, slice, c0, c1;
    slice_of(t, mt, ntile, slice, c0, c1);
    for (int r = 0; r < nt && mt * nt + r < args.M; r += kAgainRows)
      make_again<kSplitRows, kSplitThreads>(reinterpret_cast<float*>(smem), args.A, args.W, args.bias, args.out, min(args.M, (mt + 1) * nt), args.N, args.K,
                             mt * nt + r, ntile * kSplitRows);
  }
}

// C [M, N] = the slices' sums in order (+ bias): 32 rows x 64 columns a block, 4 rows a thread.
constexpr int kSumCols = 64, kSumRows = 4, kSumThreads = kSumCols * kAgainRows / kSumRows;
__global__ void __launch_bounds__(kSumThreads) split_slices_kernel(const float* __restrict__ parts, int slices, const float* __restrict__ A,
                                                                   const float* __restrict__ W, const float* __restrict__ bias, float* C,
                                                                   int M, int N, int K) {
  __shared__ __align__(16) float smem[again_floats(kSumCols)];
  const int n0 = blockIdx.x * kSumCols, m0 = blockIdx.y * kAgainRows, n = n0 + threadIdx.x % kSumCols, m = m0 + threadIdx.x / kSumCols * kSumRows;
  const int rows = n < N ? min(kSumRows, M - m) : 0;
  const size_t total = (size_t)M * N;
  const float* from = parts + (size_t)m * N + n;
  float v[kSumRows] = {};
#pragma unroll 6
  for (int s = 0; s < slices; ++s) {
#pragma unroll
    for (int r = 0; r < kSumRows; ++r)
      if (r < rows) v[r] = s == 0 ? from[(size_t)r * N] : v[r] + from[s * total + (size_t)r * N];
  }
  const float b = bias && rows > 0 ? bias[n] : 0.0f;
  bool again = false;
#pragma unroll
  for (int r = 0; r < kSumRows; ++r) {
    if (r < rows) {
      const bool lost = made_again(v[r]);
      again = again || lost;
      C[(size_t)(m + r) * N + n] = lost ? placeholder(v[r]) : bias ? v[r] + b : v[r];
    }
  }
  if (__syncthreads_or(again)) make_again<kSumCols, kSumThreads>(smem, A, W, bias, C, M, N, K, m0, n0);
}

static int split_sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 1;
  }
  return sms;
}


// Chunks of 64 k in a slice: enough slices for about one block an SM with a single tile of tokens, at least four chunks each.
// From N and K alone, so that the order of additions does not depend on the rows.
static int split_slice_chunks(int N, int K) {
  const int chunks = (K + kSplitK - 1) / kSplitK, n_tiles = (N + kSplitRows - 1) / kSplitRows;
  int slices = 148 / n_tiles;
  if (slices > chunks / 4) slices = chunks / 4;
  if (slices < 1) slices = 1;
  return (chunks + slices - 1) / slices;
}
static int split_slices(int N, int K) {
  const int per = split_slice_chunks(N, K);
  return ((K + kSplitK - 1) / kSplitK + per - 1) / per;
}

// Token rows worked on at a time: up to 1,024, fewer where their planes and slices would take more than 64 MB (18,944 -> 3,584 takes
// 185 KB a row: 256; one tile of 128 rows has a block for every SM, so that smaller portions cost launches alone).
constexpr int kSplitRowBlock = 1024;
constexpr long long kSplitScratch = 64ll << 20;
static long long split_planes(long long rows, int K) { return (rows * K * 6 + 255) / 256 * 256; }
static int split_row_block(int M, int N, int K) {
  const int slices = split_slices(N, K);
  const long long row = (long long)K * 6 + (slices > 1 ? (long long)slices * N * 4 : 0), fit = (kSplitScratch - 256) / row;
  const int most = fit >= kSplitRowBlock ? kSplitRowBlock : fit >= kSplitRows ? (int)fit / kSplitRows * kSplitRows : fit >= 16 ? (int)fit / 16 * 16 : 16;
  return M < most ? M : most;
}

template <int NT>
static int launch_split(const CUtensorMap& mw, const CUtensorMap& mt, const SplitArgs& args, size_t smem, cudaStream_t stream) {
  auto kern = gemm_f32_split_kernel<NT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int tiles = args.m_tiles * args.n_tiles * args.slices;
  kern<<<tiles < split_sm_count() ? tiles : split_sm_count(), kSplitThreads, smem, stream>>>(mw, mt, args);
  IFX_CHECK_LAUNCH();
  return 0;
}

static int make_f32_map(CUtensorMap* map, const void* base, long long rows, int cols) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return -1;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 4};
  cuuint32_t box[2] = {32u, (cuuint32_t)kSplitRows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 2000 + (int)r;
}

}  // namespace ifx

using namespace ifx;

extern "C" {

// Bytes of scratch that ifx_gemm_f32_split needs: 64 MB at most, or what 16 rows take.
long long ifx_gemm_f32_split_scratch(int M, int N, int K) {
  const long long m = split_row_block(M, N, K);
  const int slices = split_slices(N, K);
  return split_planes(m, K) + (slices > 1 ? slices * m * N * 4 : 0);
}

int ifx_gemm_f32_split_launches(int M, int N, int K) {
  const int block = split_row_block(M, N, K);
  return (M + block - 1) / block * (split_slices(N, K) > 1 ? 3 : 2);
}

// A [M, K], W [N, K], C [M, N] float32, K a multiple of 8, A, W and scratch on 16-byte boundaries.
int ifx_gemm_f32_split(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, void* scratch,
                       long long scratch_bytes, int* error_flag, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 8 || error_flag == nullptr || scratch == nullptr) return IFX_E_BADARG;
  if (((uintptr_t)A | (uintptr_t)W | (uintptr_t)scratch) % 16) return IFX_E_ALIGN;
  if (scratch_bytes < ifx_gemm_f32_split_scratch(M, N, K)) return IFX_E_TOOBIG;
  CUtensorMap mw;
  int rc = make_f32_map(&mw, W, N, K);
  if (rc) return rc;
  const int block = split_row_block(M, N, K);
  for (int r0 = 0; r0 < M; r0 += block) {
    const int m = M - r0 < block ? M - r0 : block;
    const float* a = A + (size_t)r0 * K;
    __nv_bfloat16* planes = reinterpret_cast<__nv_bfloat16*>(scratch);
    const long long n8 = (long long)m * K / 8;
    split_rows_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, stream>>>(a, planes, n8);
    IFX_CHECK_LAUNCH();
    SplitArgs args = {};
    args.A = a, args.W = W, args.bias = bias;
    args.M = m, args.N = N, args.K = K;
    args.m_tiles = (m + 127) / 128;
    args.nt = ((m + args.m_tiles - 1) / args.m_tiles + 15) / 16 * 16;             // tiles of about the same height
    args.n_tiles = (N + kSplitRows - 1) / kSplitRows;
    args.chunks = (K + kSplitK - 1) / kSplitK;
    args.slice_chunks = split_slice_chunks(N, K);
    args.slices = split_slices(N, K);
    args.w_log = args.nt <= 64 ? 2 : 1;                                            // 64: 128 + 72 KB; 128: 64 + 144 KB
    args.error_flag = error_flag;
    float* parts = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(scratch) + split_planes(m, K));
    args.out = args.slices > 1 ? parts : C + (size_t)r0 * N;
    CUtensorMap mt;
    rc = make_tensor_map_bf16(&mt, planes, 3LL * m, K, args.nt);
    if (rc) return rc;
    const size_t smem = 1024 + ((size_t)kSplitWBytes << args.w_log) + (size_t)kSplitTStages * 3 * args.nt * kSplitK * 2;
    if (args.nt <= 32) rc = launch_split<32>(mw, mt, args, smem, stream);
    else if (args.nt <= 64) rc = launch_split<64>(mw, mt, args, smem, stream);
    else rc = launch_split<128>(mw, mt, args, smem, stream);
    if (rc) return rc;
    if (args.slices > 1) {
      const dim3 grid((N + kSumCols - 1) / kSumCols, (m + kAgainRows - 1) / kAgainRows);
      split_slices_kernel<<<grid, kSumThreads, 0, stream>>>(parts, args.slices, a, W, bias, C + (size_t)r0 * N, m, N, K);
      IFX_CHECK_LAUNCH();
    }
  }
  return 0;
}

}  // extern "C"
