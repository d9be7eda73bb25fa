// The experts of a step with few tokens (decode batches, short portions) on the 5th-generation tensor cores: every expert's
// weights are read once, whatever the number of tokens that chose it, where the per-token kernels of moe.cu read an expert
// again for each of them (from L2 at best).
//
//   up     act[p] = relu(W_up[e] h[t])^2, or gated, for the (token, choice) pairs p of expert e
//   down   y[p]   = weight[p] * (W_down[e] act[p])                       float32, in slices of K where blocks are few
//   sum    out[t] = sum over the token's choices, in their order, of y[p], or weight * h[t] for an expert without weights
//
// up and down are one kernel.  A block owns 128 weight rows of one expert (gated: 64 gate rows and the 64 up rows of the
// same outputs) as the MMA's A operand and all of K; the expert's pairs, found by looking through the step's ids, are the
// MMA's N, rounded up to 16 and known only on the device.  Nothing is sorted: rows are gathered by the pair's number.
//
//   warp 0     weight tiles [128 x 64] by TMA (128-byte swizzle) into a ring of stages
//   warp 1     tcgen05.mma, tensor memory
//   warps 2-5  epilogue: activation or weight, rows of act / y
//   warp 6     the pairs' rows into the stages by cp.async, swizzled as TMA would, AHEAD stages before they are handed over
//
// An expert with more pairs than a block takes at once (`nmax`) goes through its weights again.  A step with fewer than two pairs
// an expert has blocks for as many experts as it has pairs, and the i-th of them finds the i-th expert that some token chose
// (blocks for all experts, most of which leave at once, cost 7 ns each: 110 us with 256 experts of 2,048 x 1,024).
//
// Bound: reading the chosen experts' weights.  24 tokens, 16 gated experts of 1,536 x 2,240, four a token (330 MB): the
// per-token kernels 244 us (up 146, down 98), these 81 (4.1 TB/s; 5.1 TB/s on matrices five times as large: what is lost is
// three launches' beginnings and ends).
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace ifx {

constexpr int kStreamMaxPairs = 512;          // pairs of a step
constexpr int kStreamMaxExperts = 1024;
constexpr int kStreamThreads = 224;
constexpr uint32_t kStreamWeightBytes = 128 * 128;
enum { STREAM_RELU2 = 0, STREAM_GLU = 1, STREAM_DOWN = 2 };

__device__ __forceinline__ uint64_t stream_desc(uint32_t addr) {       // K-major, 128-byte rows, 128-byte swizzle
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void stream_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void stream_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void stream_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void stream_ld16(uint32_t taddr, float (&r)[16]) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

struct StreamArgs {
  const __nv_bfloat16* src;        // up: h [T, K]; down: act [pairs, K]
  const int* ids;
  const float* weights;
  void* out;                       // up: act [pairs, N] bfloat16; down: y [pairs, N] float32
  int pairs, top, N, K, group_rows, nmax, stages, slice;               // slice: k-blocks of a block
  int experts;
  int early;                       // blocks for every expert, which fetch the first weights before it is known whether it has pairs
  float limit, slope, offset;
  int* error_flag;
};

// The place-th expert that some pair chose, -1 if there are fewer: bits of chosen experts, counted by the first warp.
__device__ __forceinline__ int chosen_expert(const int* __restrict__ ids, int pairs, int experts, int place, uint32_t* bits_s, int* found_s) {
  for (int i = threadIdx.x; i < kStreamMaxExperts / 32; i += kStreamThreads) bits_s[i] = 0u;
  if (threadIdx.x == 0) *found_s = -1;
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += kStreamThreads) {
    const int e = ids[p];
    if (e >= 0 && e < experts) atomicOr(&bits_s[e >> 5], 1u << (e & 31));
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    static_assert(kStreamMaxExperts == 32 * 32, "a lane a word");
    uint32_t word = bits_s[threadIdx.x];
    int before = __popc(word);                                         // experts in front of this lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, before, o);
      if ((int)threadIdx.x >= o) before += x;
    }
    before -= __popc(word);
    int left = place - before;
    if (left >= 0 && left < __popc(word)) {
      for (; left > 0; --left) word &= word - 1;
      *found_s = (int)threadIdx.x * 32 + __ffs(word) - 1;
    }
  }
  __syncthreads();
  return *found_s;
}

// grid (tiles of N, experts or at most as many as there are pairs, slices of K)
template <int KIND, int AHEAD>
__global__ void __launch_bounds__(kStreamThreads) moe_stream_kernel(const __grid_constant__ CUtensorMap map_w, const StreamArgs a) {
  constexpr int TILE = KIND == STREAM_GLU ? 64 : 128;                  // outputs of a block
  extern __shared__ unsigned char smem_raw[];
  __shared__ int list_s[kStreamMaxPairs];                              // this expert's pairs, in any order
  __shared__ int count_s, found_s;
  __shared__ uint32_t bits_s[kStreamMaxExperts / 32];
  __shared__ float up_rows[KIND == STREAM_GLU ? 64 : 1][17];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t stage_bytes = kStreamWeightBytes + a.nmax * 128;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)a.stages * stage_bytes);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 2 * a.stages + 2);
  const uint32_t ring = smem_addr(smem), full0 = smem_addr(bars), empty0 = full0 + 8 * a.stages, done_bar = empty0 + 8 * a.stages,
                 free_bar = done_bar + 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * TILE;
  int expert = blockIdx.y;
  const uint32_t tmem_cols = a.nmax < 32 ? 32 : a.nmax;                // nmax: a power of two

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full0 + 8 * s, 2);                                     // the weights' bytes, the gathered rows
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(done_bar, 1);
    mbar_init(free_bar, 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    count_s = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_holder)), "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const int kb0 = blockIdx.z * a.slice, kblocks = min((a.K + 63) / 64 - kb0, a.slice);   // at least one
  const int ahead = a.early ? min(a.stages, kblocks) : 0;
  auto weights = [&](int i) {                                          // k-block i of the walk into its stage
    const uint32_t dst = ring + (i % a.stages) * stage_bytes, bar = full0 + 8 * (i % a.stages);
    const int kx = (kb0 + i % kblocks) * 64, row = expert * a.group_rows + n0;
    const uint64_t policy = l2_evict_first_policy();
    mbar_expect_tx(bar, kStreamWeightBytes);
    tma_load_2d_hint(dst, &map_w, kx, row, bar, policy);
    if (KIND == STREAM_GLU) tma_load_2d_hint(dst + kStreamWeightBytes / 2, &map_w, kx, row + a.N, bar, policy);
  };
  if (threadIdx.x == 0)
    for (int i = 0; i < ahead; ++i) weights(i);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  pdl_wait();
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;
  if (!a.early) expert = chosen_expert(a.ids, a.pairs, a.experts, blockIdx.y, bits_s, &found_s);
  for (int p = threadIdx.x; p < a.pairs; p += kStreamThreads)
    if (expert >= 0 && a.ids[p] == expert) list_s[atomicAdd(&count_s, 1)] = p;        // a pair's place among the others changes no result
  __syncthreads();
  const int count = count_s;
  const int passes = (count + a.nmax - 1) / a.nmax, total = passes * kblocks;
  auto columns = [&](int pass) { return (min(a.nmax, count - pass * a.nmax) + 15) & ~15; };

  if (warp == 0) {
    // ------------------------------------------------------------ weights
    if (lane == 0) {
      bool ok = true;
      int issued = ahead;
      for (int i = ahead; i < total; ++i) {
        const int s = i % a.stages;
        if (i >= a.stages) ok = mbar_wait(empty0 + 8 * s, ((i / a.stages) & 1) ^ 1);
        if (!ok) break;
        weights(i);
        issued = i + 1;
      }
      if (!ok) {
        atomicExch(a.error_flag, 41);
        for (int i = max(0, issued - a.stages); i < issued; ++i) mbar_wait(full0 + 8 * (i % a.stages), (i / a.stages) & 1);
      }
      if (total == 0) {                                                // nothing to do after all: let what was asked for land
        for (int i = 0; i < ahead; ++i) {
          stream_arrive(full0 + 8 * i);
          if (!mbar_wait(full0 + 8 * i, 0)) atomicExch(a.error_flag, 41);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ products
    if (lane == 0) {
      bool ok = true;
      int i = 0;
      for (int pass = 0; pass < passes; ++pass) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(columns(pass) >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        if (pass > 0 && ok) ok = mbar_wait(free_bar, (pass - 1) & 1);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < kblocks && ok; ++kb, ++i) {
          const int s = i % a.stages;
          ok = mbar_wait(full0 + 8 * s, (i / a.stages) & 1);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t w_desc = stream_desc(ring + s * stage_bytes), x_desc = stream_desc(ring + s * stage_bytes + kStreamWeightBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) stream_mma(tmem_base, w_desc + 2 * k, x_desc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          stream_commit(empty0 + 8 * s);
        }
        stream_commit(done_bar);                                       // the sums are complete, or nothing more will come
      }
      if (!ok) atomicExch(a.error_flag, 42);
    }
    __syncwarp();
  } else if (warp == 6) {
    // ------------------------------------------------------------ rows of the pairs
    bool ok = true;
    for (int i = 0; i < total + AHEAD; ++i) {
      if (i < total && ok) {
        const int s = i % a.stages, pass = i / kblocks, k0 = (kb0 + i % kblocks) * 64, n = columns(pass);
        if (i >= a.stages) ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ((i / a.stages) & 1) ^ 1));
        const uint32_t dst = ring + s * stage_bytes + kStreamWeightBytes;
        const int c = lane & 7, k = k0 + c * 8;
        if (ok)
          for (int r = lane >> 3; r < n; r += 4) {
            const int at = pass * a.nmax + r;
            const bool there = at < count && k < a.K;
            const int p = list_s[min(at, count - 1)];
            const __nv_bfloat16* from = a.src + (size_t)(KIND == STREAM_DOWN ? p : p / a.top) * a.K + (there ? k : 0);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * 128 + ((c ^ (r & 7)) << 4)), "l"(from),
                         "r"(there ? 16 : 0)
                         : "memory");
          }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (!ok) break;
      if (i >= AHEAD) {
        asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD) : "memory");
        fence_proxy_async_smem();                                      // each lane's own writes, before the MMA's reads
        __syncwarp();
        if (lane == 0) stream_arrive(full0 + 8 * ((i - AHEAD) % a.stages));
      }
    }
    if (!ok && lane == 0) atomicExch(a.error_flag, 43);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else {
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3;
    const bool up_half = KIND == STREAM_GLU && quarter >= 2;           // lanes 0-63: gate rows, 64-127: up rows
    const int n = n0 + (KIND == STREAM_GLU ? (quarter & 1) * 32 : quarter * 32) + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    for (int pass = 0; pass < passes; ++pass) {
      const bool ok = mbar_wait(done_bar, pass & 1);
      if (!ok && lane == 0) atomicExch(a.error_flag, 44);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      __syncwarp();
      for (int c = 0; c < columns(pass); c += 16) {
        float v[16];
        stream_ld16(taddr + c, v);
        if (KIND == STREAM_GLU) {
          float* half = up_rows[(quarter & 1) * 32 + lane];
          if (up_half) {
#pragma unroll
            for (int j = 0; j < 16; ++j) half[j] = v[j];
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
          if (!up_half) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float gate = fminf(v[j], a.limit), up = fminf(fmaxf(half[j], -a.limit), a.limit);
              v[j] = gate / (1.0f + expf(-a.slope * gate)) * (up + a.offset);
            }
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");               // read before the next columns go over it
        }
        if (KIND == STREAM_RELU2) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.0f) * fmaxf(v[j], 0.0f);
        }
        if (n < a.N && !up_half) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int at = pass * a.nmax + c + j;
            if (at >= count) break;
            const int p = list_s[at];
            if (KIND == STREAM_DOWN) reinterpret_cast<float*>(a.out)[((size_t)blockIdx.z * a.pairs + p) * a.N + n] = v[j] * a.weights[p];
            else reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)p * a.N + n] = __float2bfloat16_rn(v[j]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) stream_arrive(free_bar);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

// grid (tokens, pieces of the width): four columns a thread.
template <typename TO>
__global__ void moe_stream_sum_kernel(const __nv_bfloat16* __restrict__ h, const float* __restrict__ y, const int* __restrict__ ids,
                                      const float* __restrict__ weights, TO* __restrict__ out, int top, int experts, int width,
                                      int slices) {
  pdl_wait();
  const int t = blockIdx.x, c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (c >= width) return;
  float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int k = 0; k < top; ++k) {
    const int p = t * top + k, e = ids[p];
    if (e >= 0 && e < experts) {
      for (int s = 0; s < slices; ++s) {
        const float4 v = *reinterpret_cast<const float4*>(y + ((size_t)s * gridDim.x * top + p) * width + c);
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
      }
    } else {
      const float w = weights[p];
      const __nv_bfloat162* x = reinterpret_cast<const __nv_bfloat162*>(h + (size_t)t * width + c);
      const float2 lo = __bfloat1622float2(x[0]), hi = __bfloat1622float2(x[1]);
      acc.x = fmaf(w, lo.x, acc.x);
      acc.y = fmaf(w, lo.y, acc.y);
      acc.z = fmaf(w, hi.x, acc.z);
      acc.w = fmaf(w, hi.y, acc.w);
    }
  }
  TO* o = out + (size_t)t * width + c;
  o[0] = from_f32<TO>(acc.x);
  o[1] = from_f32<TO>(acc.y);
  o[2] = from_f32<TO>(acc.z);
  o[3] = from_f32<TO>(acc.w);
}

template <int KIND, int AHEAD>
static int launch_stream_ahead(const CUtensorMap& mw, const StreamArgs& a, int experts, int slices, cudaStream_t stream) {
  const int tile = KIND == STREAM_GLU ? 64 : 128;
  const size_t smem = 1024 + a.stages * (kStreamWeightBytes + (size_t)a.nmax * 128) + (2 * a.stages + 2) * 8 + 16;
  auto kern = moe_stream_kernel<KIND, AHEAD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return launch_pdl(kern, dim3((a.N + tile - 1) / tile, a.early || experts < a.pairs ? experts : a.pairs, slices), dim3(kStreamThreads), smem, stream, 1, mw, a);
}

template <int KIND>
static int launch_stream(const CUtensorMap& mw, StreamArgs a, int experts, int slices, cudaStream_t stream) {
  // two blocks an SM; a row is asked for AHEAD stages early, since a read from L2 takes as long as several weight tiles
  a.stages = (int)((104 * 1024) / (kStreamWeightBytes + (size_t)a.nmax * 128));
  a.slice = ((a.K + 63) / 64 + slices - 1) / slices;
  slices = ((a.K + 63) / 64 + a.slice - 1) / a.slice;       // none of them empty
  return a.stages >= 5 ? launch_stream_ahead<KIND, 4>(mw, a, experts, slices, stream)
                       : launch_stream_ahead<KIND, 2>(mw, a, experts, slices, stream);
}

}  // namespace ifx

using namespace ifx;

extern "C" {

// Slices that the second product's K is cut into: its tiles are few and its K is long (us of the whole call, one and three slices:
// 1,536 x 2,240 gated, 1 token 57 and 47, 24 tokens 83.6 and 83.0; 3,584 x 7,104, 1 token 137 and 113, 24 tokens 355 and 341;
// six slices are slower again).
int ifx_moe_stream_slices(int ff) {
  const int kblocks = (ff + 63) / 64, want = kblocks < 12 ? 1 : 3, slice = (kblocks + want - 1) / want;
  return (kblocks + slice - 1) / slice;
}

// h [T, width], w_up [experts, ff or 2 ff (glu), width], w_down [experts, width, ff], act [T top, ff] bfloat16; y [slices, T top,
// width] float32 with as many slices as ifx_moe_stream_slices says; out [T, width] in out_dtype.  glu: as ifx_moe_experts_glu.  T top <= 512; width and ff multiples of 8; everything on
// 16-byte boundaries.
int ifx_moe_stream(const void* h, const void* w_up, const void* w_down, const int* ids, const float* weights, void* act, float* y,
                   void* out, int T, int top, int experts, int width, int ff, int out_dtype, int glu, float limit, float slope,
                   float offset, int* error_flag, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (top <= 0 || experts <= 0 || width <= 0 || ff <= 0 || error_flag == nullptr) return IFX_E_BADARG;
  if ((long long)T * top > kStreamMaxPairs || experts > kStreamMaxExperts) return IFX_E_TOOBIG;
  if (width % 8 || ff % 8 || ((uintptr_t)h | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)act | (uintptr_t)y | (uintptr_t)out) % 16)
    return IFX_E_ALIGN;
  if (out_dtype != IFX_DT_F32 && out_dtype != IFX_DT_BF16) return IFX_E_DTYPE;
  CUtensorMap mu, md;
  int rc = weight_tensor_map(&mu, w_up, (long long)experts * ff * (glu ? 2 : 1), width, glu ? 64 : 128);
  if (rc) return rc;
  rc = weight_tensor_map(&md, w_down, (long long)experts * width, ff, 128);
  if (rc) return rc;
  StreamArgs a;
  a.ids = ids;
  a.weights = weights;
  a.pairs = T * top;
  a.top = top;
  a.experts = experts;
  a.early = a.pairs >= 2 * experts;                                    // then nearly every expert has some
  a.nmax = T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : 128;           // a token chooses an expert once
  a.stages = 0;
  a.limit = limit;
  a.slope = slope;
  a.offset = offset;
  a.error_flag = error_flag;
  a.src = (const __nv_bfloat16*)h;
  a.out = act;
  a.N = ff;
  a.K = width;
  a.group_rows = glu ? 2 * ff : ff;
  rc = glu ? launch_stream<STREAM_GLU>(mu, a, experts, 1, stream) : launch_stream<STREAM_RELU2>(mu, a, experts, 1, stream);
  if (rc) return rc;
  a.src = (const __nv_bfloat16*)act;
  a.out = y;
  a.N = width;
  a.K = ff;
  a.group_rows = width;
  const int slices = ifx_moe_stream_slices(ff);
  rc = launch_stream<STREAM_DOWN>(md, a, experts, slices, stream);
  if (rc) return rc;
  const int threads = 128;
  const dim3 grid(T, (width + threads * 4 - 1) / (threads * 4));
  if (out_dtype == IFX_DT_BF16)
    return launch_pdl(moe_stream_sum_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream, 1, (const __nv_bfloat16*)h, (const float*)y,
                      ids, weights, (__nv_bfloat16*)out, top, experts, width, slices);
  return launch_pdl(moe_stream_sum_kernel<float>, grid, dim3(threads), 0, stream, 1, (const __nv_bfloat16*)h, (const float*)y, ids, weights,
                    (float*)out, top, experts, width, slices);
}

}  // extern "C"
