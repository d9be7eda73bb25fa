// C[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) on the CUDA cores, accumulating in
// float32 with one fused multiply-add per product, k ascending.
//
// This is the matrix product of the 32-bit path (its large products run in gemm_f32_split.cu)
// and it takes every M, N and K.  The additions that make one
// output element happen in an order that depends on K alone, so a row's result is
// bit-for-bit the same whatever other rows share the launch.
//
// Two kernels make the same bits.  gemm_nt_kernel takes anything.  gemm_f32_tiles_kernel takes float32 operands whose
// rows are whole 16-byte pieces: the chain of multiply-adds of an output is the same, what differs is how the
// operands arrive (cp.async, several k-blocks ahead, no pass through registers) and how many outputs a thread keeps.
#include "common.cuh"

namespace ifx {

constexpr int BM = 64, BN = 64, BK = 16, PAD = 4;

template <typename TI, typename TO>
__global__ void __launch_bounds__(256) gemm_nt_kernel(const TI* __restrict__ A, const TI* __restrict__ W,
                                                      const float* __restrict__ bias, TO* __restrict__ C,
                                                      int M, int N, int K) {
  __shared__ float As[BK][BM + PAD];
  __shared__ float Ws[BK][BN + PAD];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int lr = tid >> 2, lk = (tid & 3) * 4;

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

  const bool a_row_ok = (m0 + lr) < M, w_row_ok = (n0 + lr) < N;
  const TI* a_ptr = A + (size_t)(m0 + lr) * K;
  const TI* w_ptr = W + (size_t)(n0 + lr) * K;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + lk + i;
      As[lk + i][lr] = (a_row_ok && k < K) ? to_f32(a_ptr[k]) : 0.0f;
      Ws[lk + i][lr] = (w_row_ok && k < K) ? to_f32(w_ptr[k]) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      C[(size_t)m * N + n] = from_f32<TO>(v);
    }
  }
}

// A block makes BM x BN outputs, a thread TM x TN of them: rows ty + i (BM / TM), columns tx + j (BN / TN), a warp being
// 4 x 8 threads.  Operands stay as memory has them (k innermost), a row's BK numbers and four of padding: the eight rows
// that a quarter of a warp reads 16 bytes of at a time lie on all 32 banks once (row pitch 36 floats).  Four k steps are
// worked on per set of reads, k ascending.
// Bound: shared-memory reads beside the FMA pipe (TM + TN reads for TM TN products); 50-55 % of the pipe's rate.
// Measured (us, gemm_nt_kernel -> this): 333 rows, 1,536 -> 17,920: 861 -> 495; 8,960 -> 1,536: 655 -> 325; one row: 166 -> 34
// and 500 -> 98; 150 rows, 18,944 -> 3,584: 2,012 -> 690.
template <int BM_, int BN_, int TM, int TN, int BK_, int STAGES>
__global__ void __launch_bounds__((BM_ / TM) * (BN_ / TN)) gemm_f32_tiles_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                               const float* __restrict__ bias,
                                                                               float* __restrict__ C, int M, int N, int K) {
  constexpr int THREADS = (BM_ / TM) * (BN_ / TN), NX = BN_ / TN, NY = BM_ / TM, LD = BK_ + 4, PIECES = BK_ / 4;
  constexpr int STAGE = (BM_ + BN_) * LD;
  extern __shared__ __align__(16) float tiles[];
  constexpr int WX = NX / 8 > 0 ? NX / 8 : 1;              // warps side by side
  static_assert(NX % 8 == 0 && NY % 4 == 0, "a warp is 4 x 8 threads");
  const int tid = threadIdx.x, tx = (tid >> 5) % WX * 8 + (tid & 7), ty = (tid >> 5) / WX * 4 + ((tid >> 3) & 3);
  const int m0 = blockIdx.x * BM_, n0 = blockIdx.y * BN_;
  const int kblocks = (K + BK_ - 1) / BK_;
  auto fetch = [&](int kb) {                              // rows or k beyond the operand arrive as zeros
    float* dst = tiles + (kb % STAGES) * STAGE;
    const int k0 = kb * BK_;
#pragma unroll
    for (int e = tid; e < (BM_ + BN_) * PIECES; e += THREADS) {
      const int row = e / PIECES, k = k0 + (e % PIECES) * 4;
      const bool of_a = row < BM_;
      const int r = of_a ? m0 + row : n0 + row - BM_;
      const bool there = r < (of_a ? M : N) && k < K;
      const float* src = there ? (of_a ? A : W) + (size_t)r * K + k : A;
      const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + row * LD + (e % PIECES) * 4);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(there ? 16 : 0) : "memory");
    }
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < kblocks) fetch(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kb = 0; kb < kblocks; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                      // this block has arrived; the stage fetched next has been read by all
    if (kb + STAGES - 1 < kblocks) fetch(kb + STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* a_s = tiles + (kb % STAGES) * STAGE;
    const float* w_s = a_s + BM_ * LD;
#pragma unroll
    for (int k = 0; k < BK_; k += 4) {
      float4 a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(a_s + (ty + i * NY) * LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(w_s + (tx + j * NX) * LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * NY;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * NX;
      if (n < N) C[(size_t)m * N + n] = bias ? acc[i][j] + bias[n] : acc[i][j];
    }
  }
}

template <int BM_, int BN_, int TM, int TN, int BK_, int STAGES>
static int launch_f32_tiles(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
  auto kern = gemm_f32_tiles_kernel<BM_, BN_, TM, TN, BK_, STAGES>;
  const size_t smem = (size_t)STAGES * (BM_ + BN_) * (BK_ + 4) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  kern<<<dim3((M + BM_ - 1) / BM_, (N + BN_ - 1) / BN_), (BM_ / TM) * (BN_ / TN), smem, stream>>>(A, W, bias, C, M, N, K);
  IFX_CHECK_LAUNCH();
  return 0;
}

}  // namespace ifx

using namespace ifx;

// in_dtype: dtype of A and W.  out_dtype: dtype of C (float32 or the input dtype).
extern "C" int ifx_gemm_generic(const void* A, const void* W, const float* bias, void* C, int M, int N, int K,
                                int in_dtype, int out_dtype, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return IFX_E_BADARG;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return IFX_E_TOOBIG;
  if (in_dtype == IFX_DT_F32 && out_dtype == IFX_DT_F32 && K % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && N <= 32 * 65535) {
    // Tiles no higher than the rows there are; narrow ones where wide ones would leave SMs without a block (a block walks all
    // of K, so its chain of k steps is the time).  Measured at 1,536 columns, K 8,960: 17 rows 32 x 64 200 us, 32 x 32 151;
    // 150 rows (120 tiles of 32 x 64) 211 and 217; 16 rows 16 x 64 151, 8 x 64 99.  At 17,920 columns, K 1,536, 16 rows:
    // 16 x 64 42 us, 8 x 64 52.  64- and 128-row tiles gained nothing (333 rows: 511 and 488 against 495 us).
    const float *a = (const float*)A, *w = (const float*)W;
    float* c = (float*)C;
    const long long n_tiles = (N + 63) / 64;
    if (M <= 8 || (M <= 16 && n_tiles < 148)) return launch_f32_tiles<8, 64, 2, 2, 32, 5>(a, w, bias, c, M, N, K, stream);
    if (M <= 16) return launch_f32_tiles<16, 64, 4, 2, 32, 4>(a, w, bias, c, M, N, K, stream);
    if ((M + 31) / 32 * n_tiles >= 120) return launch_f32_tiles<32, 64, 4, 4, 32, 4>(a, w, bias, c, M, N, K, stream);
    return launch_f32_tiles<32, 32, 4, 2, 32, 4>(a, w, bias, c, M, N, K, stream);
  }
  if (in_dtype == IFX_DT_F32 && out_dtype == IFX_DT_F32)
    gemm_nt_kernel<float, float><<<grid, 256, 0, stream>>>((const float*)A, (const float*)W, bias, (float*)C, M, N, K);
  else if (in_dtype == IFX_DT_BF16 && out_dtype == IFX_DT_BF16)
    gemm_nt_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, stream>>>(
        (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, bias, (__nv_bfloat16*)C, M, N, K);
  else if (in_dtype == IFX_DT_BF16 && out_dtype == IFX_DT_F32)
    gemm_nt_kernel<__nv_bfloat16, float><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)A, (const __nv_bfloat16*)W,
                                                                   bias, (float*)C, M, N, K);
  else
    return IFX_E_DTYPE;
  IFX_CHECK_LAUNCH();
  return 0;
}
