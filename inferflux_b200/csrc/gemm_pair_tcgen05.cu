// Matrix products of pairs of SMs: 256 weight rows x up to 256 token rows a tile, on the 5th-generation tensor cores
// (tcgen05 cta_group::2), operands swapped so that the weight rows are the lanes of tensor memory and the tokens the columns.
//
// Token rows lie sorted in stretches, one per matrix of a stack (experts); a device list (PairItem) says which matrix a stretch
// takes, and cuts it into tiles of about the same width, a multiple of 32: no row is padded to 128.  Without a list all rows take
// the one matrix there is.
//
//   PAIR_RELU2  out[row, n] = max(acc, 0)^2                                        (bfloat16)
//   PAIR_F32    out[row, n] = acc, or [slices, row, n] with K in slices            (float32)
//   PAIR_GLU    the matrix holds `n` gate rows above `n` up rows; out[row, n] = g sigmoid(slope g) (u + offset) with
//               g = min(acc_gate, limit), u = clamp(acc_up, -limit, limit)         (bfloat16)
//   PAIR_GLU_EXACT  the same without the fast exponential and division
//   PAIR_SWIGLU the same without limits, slope 1 and offset 0: silu(acc_gate) acc_up, NaN included
//
// A persistent grid of one block per SM, two of them a cluster.  Both blocks load half of the weight rows and half of the tokens
// of a tile; the tensor cores of both read both halves of the tokens.  Per block:
//
//   warp 0     TMA (128-byte swizzle) of [128 weight rows x 64] and up to [128 token rows x 64] per k-block into a ring of six
//              stages.  Both blocks' copies count on the first block's barrier.
//   warp 1     (first block) tcgen05.mma M 256, N, K 16 into one of two accumulators; commits free the stage in both blocks
//   warps 2-5  epilogue of this block's 128 weight rows, under the products of the next tile
//
// Gate and up rows of one output lie in one warp's lanes, `half_rows` (8 or 16) apart: the tensor map interleaves them.
//
// Why pairs: an SM takes operands in at 64 bytes a cycle.  A block alone, 128 x 256, needs 48 KB per 64 k, 768 cycles of it for
// 512 of the tensor pipe; a block of a pair needs 32 KB.  Tiles in bands: blocks running at a time share few matrices, each of
// which is read from memory once.
// A stage is two copies, one a matrix: five (tokens in boxes of 32 rows) took a tenth longer.  8,192 rows of 4,096 against two
// matrices of 4,096: 170 us, 1.62 PFLOP/s, the library's best; with few tiles what is lost is the last wave (192 tiles on 74 pairs).
// Measured, all kernels of a mixture of 16 experts, four a token, 128 x 256 tiles of single blocks with rows padded to 128 (few
// tokens: a stream of single blocks that gathered each expert's pairs) -> this (us): 2,048 tokens, 1,536 x 3,328: 260 -> 208;
// 24 tokens, 1,536 x 2,240 gated: 98 -> 80; 700 tokens, 3,584 x 4,736 gated: 478 -> 362.
//
// One matrix: 1,531 rows, 1,536 -> 2 x 8,960: 65 -> 59; 4,096, 3,584 -> 2 x 18,944: 811 -> 675 (1.65 PFLOP/s).
//
// No load has a multicast form; the commits that arrive at both blocks' barriers do.  Every wait on an mbarrier is bounded.  Two waits
// are not: the cluster's barriers, which both blocks reach whatever their waits came to, and tcgen05.alloc, which waits for what
// another kernel's blocks still hold on the SM.
#include "common.cuh"
#include "ptx_sm100.cuh"
#include "moe_items.cuh"

namespace ifx {

constexpr int kPairRows = 256, kPairTokens = 256, kPairK = 64, kPairStages = 6;   // weight rows and tokens of a tile, k of a stage
constexpr uint32_t kPairWBytes = 128 * kPairK * 2, kPairStageBytes = 2 * kPairWBytes;
constexpr int kPairThreads = 192;
enum { PAIR_RELU2 = 0, PAIR_F32 = 1, PAIR_GLU = 2, PAIR_SWIGLU = 3, PAIR_GLU_EXACT = 4 };

// The token rows in boxes of 32, 64 and 128: a block's share of a tile is one copy.
struct TokenMaps {
  CUtensorMap rows[3];
};

struct PairArgs {
  const PairItem* items;             // items[0].matrix: how many follow; null: `rows` rows in `row_tiles` tiles
  int rows, row_tiles;
  void* out;
  int N, kblocks, w_tiles, half_rows, band;
  int slices, slice_kblocks;         // PAIR_F32: K in slices, each with its own [rows, N] of `out`
  float limit, slope, offset;
  int* error_flag;
};

__device__ __forceinline__ uint64_t pair_desc(uint32_t addr) {         // K-major, 128-byte rows, 128-byte swizzle
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// mbar_wait with a limit in time instead of tries (half a second): a stalled pair ends soon, whatever a try takes.
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity) {
  uint64_t begin = 0;
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    uint64_t now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (begin == 0) begin = now;
    if (now - begin > 500000000ull) return false;
  }
}
__device__ __forceinline__ uint32_t pair_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t pair_first_blocks(uint32_t addr) { // the same place in the first block's shared memory
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void pair_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void pair_load_5d(uint32_t dst, const CUtensorMap* map, int x, int block, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(0), "r"(block), "r"(z) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}
__device__ __forceinline__ void pair_commit(uint32_t bar, uint32_t elected) {     // arrives at both blocks' barrier
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t}"
      ::"r"(bar), "r"(elected), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void pair_arrive_at_first(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(pair_first_blocks(bar)) : "memory");
}
__device__ __forceinline__ void pair_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t pair_pack(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Tile i of `tiles` that share `rows` rows: sizes differ by one at most.
__device__ __forceinline__ PairItem even_share(int rows, int tiles, int i) {
  const int base = rows / tiles, more = rows % tiles, n = base + (i < more);
  return PairItem{0, i * base + min(i, more), n, (n + 31) / 32 * 32};
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ TokenMaps map_t, const PairArgs args) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bars[2 * kPairStages + 4];
  __shared__ uint32_t tmem_holder;
  // both blocks' stages must lie at the same place: the shared window's own address is aligned, not the generic one
  const uint32_t ring = (smem_addr(smem_raw) + 1023) & ~1023u;
  const uint32_t full = smem_addr(bars), empty = full + 8 * kPairStages, acc_full = empty + 8 * kPairStages, acc_empty = acc_full + 16;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = (int)pair_rank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Tensor memory of a pair is taken and given back by both blocks together.  So a block asks for it only once it knows that the
  // other one runs (with programmatic launch it may have started where a block of the kernel before has only just left), and
  // leaves only behind the other's return.
  __syncthreads();
  pair_sync();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pair_sync();
  const uint32_t tmem = tmem_holder;
  pdl_wait();

  const int items = args.items ? args.items[0].matrix : args.row_tiles, tiles = items * args.w_tiles * (MODE == PAIR_F32 ? args.slices : 1), pairs = gridDim.x >> 1;
  // Bands of `band` items with all their weight tiles: slices of K fastest, then items.
  auto tile_at = [&](int t, PairItem& item, int& wt, int& slice) {
    slice = 0;
    if (MODE == PAIR_F32) {
      slice = t % args.slices;
      t /= args.slices;
    }
    const int first = t / (args.band * args.w_tiles) * args.band, rows = min(args.band, items - first), in = t - first * args.w_tiles;
    item = args.items ? args.items[1 + first + in % rows] : even_share(args.rows, items, first + in % rows);
    wt = in / rows;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    if (lane == 0) {
      const uint32_t full_first = pair_first_blocks(full);
      int idx = 0;
      bool ok = true;
      for (int t = blockIdx.x >> 1; t < tiles && ok; t += pairs) {
        PairItem item;
        int wt, slice;
        tile_at(t, item, wt, slice);
        const int kb0 = slice * args.slice_kblocks, kb1 = min(args.kblocks, kb0 + args.slice_kblocks);
        const int half = item.width / 2, box = half <= 32 ? 0 : (half <= 64 ? 1 : 2);
        const uint32_t bytes = kPairWBytes + (32u << box) * kPairK * 2;
        for (int kb = kb0; kb < kb1; ++kb, ++idx) {
          const int s = idx % kPairStages;
          if (idx >= kPairStages) ok = pair_wait(empty + 8 * s, ((idx / kPairStages) & 1) ^ 1);
          if (!ok) break;
          if (rank == 0) mbar_expect_tx(full + 8 * s, 2 * bytes);
          const uint32_t dst = ring + s * kPairStageBytes, bar = full_first + 8 * s;
          if (MODE >= PAIR_GLU) pair_load_5d(dst, &map_w, kb * kPairK, (wt * 128 + rank * 64) / args.half_rows, item.matrix, bar);
          else pair_load_3d(dst, &map_w, kb * kPairK, wt * kPairRows + rank * 128, item.matrix, bar);
          pair_load_2d(dst + kPairWBytes, &map_t.rows[box], kb * kPairK, item.row + rank * half, bar);
        }
      }
      // the commits that free the last stages arrive here too: not at a block that has left
      for (int i = max(0, idx - kPairStages); i < idx && ok; ++i) ok = pair_wait(empty + 8 * (i % kPairStages), (i / kPairStages) & 1);
      if (!ok) {                                     // copies in flight end before the block does
        atomicExch(args.error_flag, 71);
        if (rank == 0)
          for (int i = max(0, idx - kPairStages); i < idx; ++i) pair_wait(full + 8 * (i % kPairStages), (i / kPairStages) & 1);
        else
          for (int i = 0; i < 10; ++i) __nanosleep(1000000);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ products, by the first block's warp in step
    if (rank == 0) {
      const uint32_t elected = elect_one();
      int idx = 0, tile = 0;
      bool ok = true;
      for (int t = blockIdx.x >> 1; t < tiles && ok; t += pairs, ++tile) {
        PairItem item;
        int wt, slice;
        tile_at(t, item, wt, slice);
        const int kb0 = slice * args.slice_kblocks, kb1 = min(args.kblocks, kb0 + args.slice_kblocks);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(item.width >> 3) << 17) | ((uint32_t)(kPairRows >> 4) << 24);
        const int buf = tile & 1, use = tile >> 1;
        if (use > 0) ok = pair_wait(acc_empty + 8 * buf, (use & 1) ^ 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + buf * kPairTokens;
        for (int kb = kb0; kb < kb1; ++kb, ++idx) {
          const int s = idx % kPairStages;
          ok = pair_wait(full + 8 * s, (idx / kPairStages) & 1);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t a = pair_desc(ring + s * kPairStageBytes), b = pair_desc(ring + s * kPairStageBytes + kPairWBytes);
#pragma unroll
          for (int k = 0; k < kPairK / 16; ++k) pair_mma(acc, a + 2 * k, b + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u, elected);
          pair_commit(empty + 8 * s, elected);
        }
        if (ok) pair_commit(acc_full + 8 * buf, elected);
      }
      for (int i = max(0, tile - 2); i < tile && ok; ++i) ok = pair_wait(acc_empty + 8 * (i & 1), (i >> 1) & 1);   // the other block's arrivals
      if (!ok && lane == 0) atomicExch(args.error_flag, 72);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3;
    int tile = 0;
    bool ok = true;
    for (int t = blockIdx.x >> 1; t < tiles && ok; t += pairs, ++tile) {
      const int buf = tile & 1, use = tile >> 1;
      PairItem item;
      int wt, slice;
      tile_at(t, item, wt, slice);
      ok = pair_wait(acc_full + 8 * buf, use & 1);
      if (!ok) {
        if (lane == 0) atomicExch(args.error_flag, 73);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + buf * kPairTokens;
      for (int c = 0; c < item.count; c += 16) {
        float v[16];
        pair_ld16(taddr + c, v);
        const size_t row = (size_t)item.row + c;
        const int left = item.count - c;             // columns that are somebody's
        if (MODE == PAIR_F32) {
          const int n = wt * kPairRows + rank * 128 + quarter * 32 + lane;
          float* out = reinterpret_cast<float*>(args.out) + ((size_t)slice * args.rows + row) * args.N + n;
          if (n < args.N) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (j < left) out[(size_t)j * args.N] = v[j];
          }
        } else if (MODE == PAIR_RELU2) {
          // even lanes take both neighbours' outputs of column j, odd ones those of j + 1: 4-byte stores
          const int n = wt * kPairRows + rank * 128 + quarter * 32 + (lane & ~1), odd = lane & 1;
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(args.out) + row * args.N + n;
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.0f) * fmaxf(v[j], 0.0f);
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float other = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
            const uint32_t both = odd ? pair_pack(other, v[j + 1]) : pair_pack(v[j], other);
            if (n < args.N && j + odd < left) *reinterpret_cast<uint32_t*>(out + (size_t)(j + odd) * args.N) = both;
          }
        } else {
          // A gate lane makes the output of columns j, j + 2, its up lane those of j + 1, j + 3; then as above over neighbours.
          const int half = args.half_rows, up = (lane & half) != 0, odd = lane & 1;
          const int place = half == 16 ? lane & 15 : (lane >> 4) * 8 + (lane & 7);
          const int n = wt * 128 + rank * 64 + quarter * 16 + (place & ~1);
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(args.out) + row * args.N + n;
          auto made = [&](float lo, float hi) {        // of columns j (lo) and j + 1 (hi)
            const float other = __shfl_xor_sync(0xffffffffu, up ? lo : hi, half);
            if (MODE == PAIR_SWIGLU) {
              const float gate = up ? other : lo;
              return __fdividef(gate, 1.0f + __expf(-gate)) * (up ? hi : other);
            }
            const float gate = fminf(up ? other : lo, args.limit), u = fminf(fmaxf(up ? hi : other, -args.limit), args.limit);
            if (MODE == PAIR_GLU_EXACT) return gate / (1.0f + expf(-args.slope * gate)) * (u + args.offset);
            return __fdividef(gate, 1.0f + __expf(-args.slope * gate)) * (u + args.offset);
          };
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            const float r01 = made(v[j], v[j + 1]), r23 = made(v[j + 2], v[j + 3]);
            const float other = __shfl_xor_sync(0xffffffffu, odd ? r01 : r23, 1);
            const uint32_t both = odd ? pair_pack(other, r23) : pair_pack(r01, other);
            const int col = j + up + 2 * odd;
            if (n < args.N && col < left) *reinterpret_cast<uint32_t*>(out + (size_t)col * args.N) = both;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) pair_arrive_at_first(acc_empty + 8 * buf);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  pair_sync();                                       // nothing arrives at, or reads from, a block that has left
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  __syncthreads();
  pair_sync();
}

static int pair_sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 2;
  }
  return sms;
}

static int pair_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return -1;
  if (reinterpret_cast<uintptr_t>(base) & 15) return IFX_E_ALIGN;
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 2000 + (int)r;
}

template <int MODE>
static int launch_pair(const CUtensorMap& mw, const TokenMaps& mt, PairArgs args, int most_items, cudaStream_t stream) {
  const size_t smem = 1024 + (size_t)kPairStages * kPairStageBytes;
  cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const long long tiles = (long long)most_items * args.w_tiles * args.slices;
  const int most = pair_sm_count() / 2, pairs = tiles < most ? (int)tiles : most;
  args.band = args.items ? (pairs + args.w_tiles - 1) / args.w_tiles : most_items;     // one matrix: all tokens against a tile of it
  return launch_pdl(gemm_pair_kernel<MODE>, dim3(2 * pairs), dim3(kPairThreads), smem, stream, 1, mw, mt, args);
}

// tokens [rows, K] bfloat16 sorted in stretches; W: `stack` matrices of [N, K] (GLU: [2 N, K]) bfloat16; K and N multiples of 8;
// items on the device, at most `most_items` of them.  slice_kblocks: 64s of K in a slice (0: all; PAIR_F32 then fills [slices, rows, N]).
int gemm_pair(int mode, const void* tokens, const void* W, void* out, int rows, int N, int K, int stack, const PairItem* items,
              int most_items, int slice_kblocks, float limit, float slope, float offset, int* error_flag, cudaStream_t stream) {
  if (rows <= 0 || N <= 0 || most_items <= 0) return 0;
  if (K <= 0 || K % 8 || N % 8 || stack <= 0 || slice_kblocks < 0 || (slice_kblocks && mode != PAIR_F32)) return IFX_E_BADARG;
  CUtensorMap mw;
  TokenMaps mt;
  const cuuint64_t k = (cuuint64_t)K, pitch = k * 2;
  PairArgs args = {};
  args.items = items, args.rows = rows, args.row_tiles = most_items, args.out = out, args.N = N, args.kblocks = (K + kPairK - 1) / kPairK;
  args.slice_kblocks = slice_kblocks ? slice_kblocks : args.kblocks;
  args.slices = (args.kblocks + args.slice_kblocks - 1) / args.slice_kblocks;
  args.limit = limit, args.slope = slope, args.offset = offset, args.error_flag = error_flag;
  int rc;
  if (mode >= PAIR_GLU) {
    args.half_rows = N % 16 ? 8 : 16;
    args.w_tiles = (N + 127) / 128;
    const cuuint64_t h = (cuuint64_t)args.half_rows;
    const cuuint64_t dims[5] = {k, h, 2, (cuuint64_t)N / h, (cuuint64_t)stack}, strides[4] = {pitch, N * pitch, h * pitch, 2 * N * pitch};
    const cuuint32_t box[5] = {kPairK, (cuuint32_t)h, 2, (cuuint32_t)(64 / h), 1};
    rc = pair_map(&mw, W, 5, dims, strides, box);
  } else {
    args.w_tiles = (N + kPairRows - 1) / kPairRows;
    const cuuint64_t dims[3] = {k, (cuuint64_t)N, (cuuint64_t)stack}, strides[2] = {pitch, N * pitch};
    const cuuint32_t box[3] = {kPairK, 128, 1};
    rc = pair_map(&mw, W, 3, dims, strides, box);
  }
  if (rc) return rc;
  const cuuint64_t dims[2] = {k, (cuuint64_t)rows}, strides[1] = {pitch};
  for (int i = 0; i < 3; ++i) {
    const cuuint32_t box[2] = {kPairK, 32u << i};
    rc = pair_map(&mt.rows[i], tokens, 2, dims, strides, box);
    if (rc) return rc;
  }
  if (mode == PAIR_RELU2) return launch_pair<PAIR_RELU2>(mw, mt, args, most_items, stream);
  if (mode == PAIR_F32) return launch_pair<PAIR_F32>(mw, mt, args, most_items, stream);
  if (mode == PAIR_GLU) return launch_pair<PAIR_GLU>(mw, mt, args, most_items, stream);
  if (mode == PAIR_GLU_EXACT) return launch_pair<PAIR_GLU_EXACT>(mw, mt, args, most_items, stream);
  if (mode == PAIR_SWIGLU) return launch_pair<PAIR_SWIGLU>(mw, mt, args, most_items, stream);
  return IFX_E_BADARG;
}

// The same for rows that all take the one matrix W.
int gemm_pair_rows(int mode, const void* tokens, const void* W, void* out, int rows, int N, int K, int* error_flag, cudaStream_t stream) {
  return gemm_pair(mode, tokens, W, out, rows, N, K, 1, nullptr, (rows + kItemTokens - 1) / kItemTokens, 0, 0.0f, 0.0f, 0.0f, error_flag,
                   stream);
}

}  // namespace ifx
