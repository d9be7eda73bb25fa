// Float32 matrix product C[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) on the 5th-generation tensor cores, at 32-bit precision.
//
// Every operand is cut into three bfloat16 numbers that add up to it exactly (24 = 8 + 8 + 8 bits: the upper 16 bits of the
// number, of what is left, and of what is left then), and an output is the sum of the six products of parts that reach 2^-16 of
// it: hi hi, hi mid, mid hi, mid mid, hi lo, lo hi.  What is left out is below 2^-23 of a product's size.  The tensor cores cut
// off when they add, so a chunk of 64 k gets an accumulator of its own, small products first, and the chunks' sums are added up
// in registers with rounded float32 additions, k ascending: fewer roundings than a chain of K multiply-adds.  Errors against 64
// bits (2-norm, normal rows; the same for 1 to 1,000 of them): K 1,536 chain of multiply-adds 7.0e-7, this 1.5e-7; K 3,584
// 10.7e-7 and 1.9e-7; K 8,960 16.9e-7 and 1.6e-7; K 18,944 24.7e-7 and 1.9e-7.
//
// An output's additions depend on K and N alone (how K is cut into slices does), never on the number of rows, so a row's bits
// are the same whatever other rows share the launch.  A result that is not finite, or is tiny enough for a part to have fallen
// below bfloat16's range, is made again as the plain chain of multiply-adds: infinities, NaN and overflow behave as there (a sum that leaves float32's range and
// returns within one chunk stays finite here).
//
// Swapped operands: 128 weight rows are the lanes of tensor memory, up to 128 token rows the columns.  Persistent blocks:
//
//   warp 0        TMA: weights as they are (float32, [128 x 64] a chunk), the tokens' three planes (split_rows_kernel) as bfloat16
//   warps 2-9     cut a chunk's weight rows, read from shared memory, and store the three parts into tensor memory (the products'
//                 A operand); four warps the even chunks, four the odd ones (one group of four: 121 us instead of 109)
//   warp 1        24 tcgen05.mma a chunk (M 128, N tokens, K 16, A from tensor memory) into one of two accumulators
//   warps 10-17   add a finished chunk's accumulator to their registers, half the columns each four; behind the last chunk store,
//                 neighbouring lanes neighbouring columns of a row
//
// Bound: the tensor pipe for many rows (1,000 rows of 3,584 -> 37,888: 1,313 us, six products at 1.24 PFLOP/s); cutting and
// reading the weights for few.  Measured, gemm_f32_tiles_kernel -> this with both kernels beside it (us): 333 rows, 1,536 ->
// 17,920: 485 -> 109; 8,960 -> 1,536: 310 -> 79; one row: 33 -> 32 and 107 -> 25; 150 rows, 18,944 -> 3,584: 650 -> 143.
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace ifx {

constexpr int kSplitRows = 128, kSplitK = 64;                    // weight rows of a tile, k of a chunk
constexpr uint32_t kSplitWBytes = kSplitRows * kSplitK * 4;      // a chunk of float32 weights
constexpr int kSplitMaxStages = 4;
constexpr int kSplitThreads = 576;
constexpr int kSplitPartCols = kSplitK / 2;                      // tensor memory columns of one part of a chunk
constexpr int kSplitACols = 3 * kSplitPartCols;

// Upper 16 bits of two numbers as a pair of bfloat16 (a below, b above).
__device__ __forceinline__ uint32_t upper_halves(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ float upper_part(float a) { return __uint_as_float(__float_as_uint(a) & 0xffff0000u); }

// a, b -> three pairs of bfloat16.  What is not finite leaves NaN in the lower parts; the result is then made again.
__device__ __forceinline__ void cut_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = upper_halves(a, b);
  const float ra = a - upper_part(a), rb = b - upper_part(b);
  mid = upper_halves(ra, rb);
  lo = upper_halves(ra - upper_part(ra), rb - upper_part(rb));
}

// planes [3, rows, K] bfloat16 <- x [rows, K] float32, eight numbers a thread.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ planes, long long n8) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= n8) return;
  const float4 a = reinterpret_cast<const float4*>(x)[2 * i], b = reinterpret_cast<const float4*>(x)[2 * i + 1];
  uint4 hi, mid, lo;
  cut_pair(a.x, a.y, hi.x, mid.x, lo.x);
  cut_pair(a.z, a.w, hi.y, mid.y, lo.y);
  cut_pair(b.x, b.y, hi.z, mid.z, lo.z);
  cut_pair(b.z, b.w, hi.w, mid.w, lo.w);
  uint4* out = reinterpret_cast<uint4*>(planes);
  out[i] = hi;
  out[n8 + i] = mid;
  out[2 * n8 + i] = lo;
}

// Whether a result has to be made again (see the top).  2^-100: parts of a number above 2^-109 are whole.
__device__ __forceinline__ bool made_again(float v) { return !(fabsf(v) < INFINITY) || (v != 0.0f && fabsf(v) < 7.9e-31f); }
__device__ __noinline__ float chain_of_products(const float* __restrict__ a, const float* __restrict__ w, int K) {
  float acc = 0.0f;
  for (int k = 0; k < K; k += 4) {
    const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
    acc = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, acc))));
  }
  return acc;
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
  int M, N, K, m_tiles, n_tiles, slices, slice_chunks, chunks, nt, w_stages, t_stages;
  int* error_flag;
};

// NT: registers for sums (token rows of a tile at most); args.nt of them are there.
template <int NT>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_t, const SplitArgs args) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bars[4 * kSplitMaxStages + 6];
  __shared__ uint32_t tmem_holder;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int nt = args.nt, w_stages = args.w_stages, t_stages = args.t_stages;
  const uint32_t plane_bytes = (uint32_t)nt * kSplitK * 2, t_bytes = 3 * plane_bytes;
  const uint32_t w_smem = smem_addr(smem), t_smem = w_smem + w_stages * kSplitWBytes;
  const uint32_t w_full = smem_addr(bars), w_empty = w_full + 8 * kSplitMaxStages, t_full = w_empty + 8 * kSplitMaxStages,
                 t_empty = t_full + 8 * kSplitMaxStages, a_full = t_empty + 8 * kSplitMaxStages, done = a_full + 16, acc_empty = done + 16;
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
      mbar_init(done + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, 8);
    }
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
  const uint32_t a_tmem = tmem + 256;                              // accumulators: columns 0 and 128; parts: 256 and 352

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
          const int ws = i % w_stages, ts = i % t_stages;
          if (i >= w_stages) ok = mbar_wait(w_empty + 8 * ws, ((i / w_stages) & 1) ^ 1);
          if (!ok) break;
          mbar_expect_tx(w_full + 8 * ws, kSplitWBytes);
          const uint32_t dst = w_smem + ws * kSplitWBytes;
          tma_load_2d(dst, &map_w, c * kSplitK, ntile * kSplitRows, w_full + 8 * ws);
          tma_load_2d(dst + kSplitWBytes / 2, &map_w, c * kSplitK + 32, ntile * kSplitRows, w_full + 8 * ws);
          if (i >= t_stages) ok = mbar_wait(t_empty + 8 * ts, ((i / t_stages) & 1) ^ 1);
          if (!ok) {
            mbar_wait(w_full + 8 * ws, (i / w_stages) & 1);        // not counted below: it has no tokens
            break;
          }
          mbar_expect_tx(t_full + 8 * ts, t_bytes);
          for (int p = 0; p < 3; ++p)
            tma_load_2d(t_smem + ts * t_bytes + p * plane_bytes, &map_t, c * kSplitK, p * args.M + mt * nt, t_full + 8 * ts);
        }
      }
      if (!ok) {
        atomicExch(args.error_flag, 61);
        for (int j = max(0, i - w_stages); j < i; ++j) mbar_wait(w_full + 8 * (j % w_stages), (j / w_stages) & 1);
        for (int j = max(0, i - t_stages); j < i; ++j) mbar_wait(t_full + 8 * (j % t_stages), (j / t_stages) & 1);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ products
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(kSplitRows >> 4) << 24);
    const uint32_t elected = elect_one();
    const uint64_t plane_step = plane_bytes >> 4;
    int i = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int mt, ntile, slice, c0, c1;
      slice_of(t, mt, ntile, slice, c0, c1);
      for (int c = c0; c < c1; ++c, ++i) {
        const int buf = i & 1, ts = i % t_stages;
        ok = mbar_wait(t_full + 8 * ts, (i / t_stages) & 1) && mbar_wait(a_full + 8 * buf, (i >> 1) & 1);
        if (ok && i >= 2) ok = mbar_wait(acc_empty + 8 * buf, ((i >> 1) & 1) ^ 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + buf * 128, a = a_tmem + buf * kSplitACols;
        const uint64_t b = split_smem_desc(t_smem + ts * t_bytes);
        // (part of the weights, part of the tokens): 0 hi, 1 mid, 2 lo; the smallest products first
        constexpr int WP[6] = {2, 0, 1, 1, 0, 0}, TP[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int k = 0; k < kSplitK / 16; ++k)
            umma_ts(acc, a + WP[p] * kSplitPartCols + k * 8, b + TP[p] * plane_step + 2 * k, idesc, (p > 0 || k > 0) ? 1u : 0u, elected);
        umma_commit(t_empty + 8 * ts, elected);
        umma_commit(done + 8 * buf, elected);
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
        const int buf = i & 1, ws = i % w_stages;
        if (buf != group) continue;
        ok = mbar_wait(w_full + 8 * ws, (i / w_stages) & 1);
        if (ok && i >= 2) ok = mbar_wait(done + 8 * buf, ((i >> 1) & 1) ^ 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t base = a_tmem + ((uint32_t)((warp & 3) * 32) << 16) + buf * kSplitACols;
#pragma unroll
        for (int h = 0; h < 2; ++h) {                              // 32 k: a row of 128 bytes, 16-byte pieces swizzled
          const unsigned char* src = smem + (size_t)ws * kSplitWBytes + h * (kSplitWBytes / 2) + row * 128;
          uint32_t hi[16], mid[16], lo[16];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 v = *reinterpret_cast<const float4*>(src + ((q ^ (row & 7)) << 4));
            cut_pair(v.x, v.y, hi[2 * q], mid[2 * q], lo[2 * q]);
            cut_pair(v.z, v.w, hi[2 * q + 1], mid[2 * q + 1], lo[2 * q + 1]);
          }
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
    int i = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      int mt, ntile, slice, c0, c1;
      slice_of(t, mt, ntile, slice, c0, c1);
      float sum[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) sum[j] = 0.0f;
      for (int c = c0; c < c1; ++c, ++i) {
        const int buf = i & 1;
        ok = mbar_wait(done + 8 * buf, (i >> 1) & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + buf * 128 + first;
#pragma unroll
        for (int j0 = 0; j0 < COLS; j0 += 16) {
          if (first + j0 < nt) {
            uint32_t r[16];
            split_tmem_ld16(taddr + j0, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j0 + j] += __uint_as_float(r[j]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) split_arrive(acc_empty + 8 * buf);
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
            again = again || made_again(sum[j]);
            out[(size_t)(m0 + j) * args.N] = sum[j] + b;
          }
        }
        if (whole && again) {                                      // rare: which of them they were is seen from the results
          for (int j = 0; j < cols; ++j)
            if (made_again(out[(size_t)(m0 + j) * args.N] - b))
              out[(size_t)(m0 + j) * args.N] = chain_of_products(args.A + (size_t)(m0 + j) * args.K, args.W + (size_t)n * args.K, args.K) + b;
        }
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
}

// C [M, N] = the slices' sums in order (+ bias).
__global__ void __launch_bounds__(256) split_slices_kernel(const float* __restrict__ parts, int slices, const float* __restrict__ A,
                                                           const float* __restrict__ W, const float* __restrict__ bias,
                                                           float* __restrict__ C, int M, int N, int K) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x, total = (long long)M * N;
  if (i >= total) return;
  float v = parts[i];
#pragma unroll 4
  for (int s = 1; s < slices; ++s) v += parts[s * total + i];
  const int n = (int)(i % N);
  if (made_again(v)) v = chain_of_products(A + i / N * K, W + (size_t)n * K, K);
  C[i] = bias ? v + bias[n] : v;
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

constexpr int kSplitRowBlock = 1024;         // token rows worked on at a time: bounds the scratch

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

// Bytes of scratch that ifx_gemm_f32_split needs.
long long ifx_gemm_f32_split_scratch(int M, int N, int K) {
  const long long m = M < kSplitRowBlock ? M : kSplitRowBlock;
  const int slices = split_slices(N, K);
  return ((m * K * 6 + 255) / 256) * 256 + (slices > 1 ? slices * m * N * 4 : 0);
}

int ifx_gemm_f32_split_launches(int M, int N, int K) {
  return (M + kSplitRowBlock - 1) / kSplitRowBlock * (split_slices(N, K) > 1 ? 3 : 2);
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
  for (int r0 = 0; r0 < M; r0 += kSplitRowBlock) {
    const int m = M - r0 < kSplitRowBlock ? M - r0 : kSplitRowBlock;
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
    args.w_stages = args.nt <= 64 ? 4 : 2;                                         // 64: 128 + 72 KB; 128: 64 + 144 KB
    args.t_stages = 3;
    args.error_flag = error_flag;
    float* parts = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(scratch) + ((long long)m * K * 6 + 255) / 256 * 256);
    args.out = args.slices > 1 ? parts : C + (size_t)r0 * N;
    CUtensorMap mt;
    rc = make_tensor_map_bf16(&mt, planes, 3LL * m, K, args.nt);
    if (rc) return rc;
    const size_t smem = 1024 + (size_t)args.w_stages * kSplitWBytes + (size_t)args.t_stages * 3 * args.nt * kSplitK * 2;
    if (args.nt <= 32) rc = launch_split<32>(mw, mt, args, smem, stream);
    else if (args.nt <= 64) rc = launch_split<64>(mw, mt, args, smem, stream);
    else rc = launch_split<128>(mw, mt, args, smem, stream);
    if (rc) return rc;
    if (args.slices > 1) {
      const long long total = (long long)m * N;
      split_slices_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(parts, args.slices, a, W, bias, C + (size_t)r0 * N, m, N, K);
      IFX_CHECK_LAUNCH();
    }
  }
  return 0;
}

}  // extern "C"
