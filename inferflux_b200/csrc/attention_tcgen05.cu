// Attention of prompt portions on the 5th-generation tensor cores.
//
// A block of the grid is up to 256 query tokens of one query head, as two tiles of 128; it
// walks the keys they may see in tiles of 128; both query tiles use each key/value tile that
// is fetched, which halves the traffic from L2.  Tensor memory holds, per query tile, the
// scores and the output:
//
//   S = Q . K^T     tcgen05.mma, M 128 (queries = TMEM lanes) x N 128 (keys), K = head size;
//                   Q and the key tile are K-major in shared memory (128-byte swizzle)
//   softmax         one group of four warps per query tile, one thread per query row: the row
//                   of S is read from TMEM once (tcgen05.ld), masked on edge tiles, exponentiated
//                   against the row's reference maximum (log2 domain, one FFMA + one ex2 per
//                   score), and written back over S as bfloat16 pairs (tcgen05.st): the A
//                   operand of the next product
//   O += P . V      tcgen05.mma with A from tensor memory; V stays as the cache holds it
//                   (key-major rows), i.e. an MN-major B operand.  O accumulates in TMEM.
//
// The MMA warp alternates between the two query tiles, so that the tensor cores work on one
// tile while the other tile's softmax runs.  A reference maximum moves only when the running
// maximum has outgrown it by more than 2^8; then the thread rescales its row of O in TMEM.
// Probabilities therefore stay below 2^8, and sum and output are taken against the same
// reference, so the result is the softmax exactly (up to rounding).
//
// Warp 0 fetches: the query tiles once, then per key tile the pages of K and of V as TMA boxes
// [16 keys x 64 elements] through the block table, into a ring of slots (a slot holds the keys
// or the values of one tile).  Warp 1 issues the MMAs.  Warps 4-7 and 8-11 are the softmax groups, with 208 registers a thread
// (setmaxnreg), since a row's scores take 128.
//
// A block has an SM to itself.  When its last keys are on their way it takes a block that has not begun off the grid
// (clusterlaunchcontrol) and goes on with that one: its keys and, once the output rows that lay in their place have left, its queries
// are fetched while the last tile's softmax and the output are still at work.  A block of its own would begin 5 us later (exit, launch
// 0.7, barriers, tensor memory, tile, slot, page and keys one after the other 2.7).  A grid of no more than 148 blocks takes none.
// The output leaves through shared memory in whole rows (a thread's own row, 16 bytes of 32 rows a store, took 2 us a tile).
//
// Bound: the tensor pipe: a key tile takes a block 1.87 us at the 1.65 GHz that the SMs keep under it, 1.3 PFLOP/s while a block
// walks its keys; the rest is heads and tails of blocks.  Blocks behind one another, whole rows of output, registers for the scores
// and two scores an instruction, us: 2,500 tokens of 28 heads behind 4,000 153 -> 139, behind none 61 -> 55; 2,200 in five prompts
// 38.5 -> 31.3; 900 of 12 heads behind 1,500 (one round) 20.5 -> 18.3, eight layers of 1,531 in three prompts 146 -> 127.  A quarter of
// the exponentials by multiply-adds was slower (149 -> 153), probabilities of the first 96 keys instead of 64 handed over first the same,
// sums of probabilities two an instruction in another order 2 % faster.
// A warp in step issues the products, one lane of it by predicate: with a single thread in a
// branch of its own a product took 108 clocks to issue instead of 65 (2,500 tokens behind 4,000, 28 heads: 211 us, then 192).
// Scores of a tile at an edge (the diagonal, a window's end, kept keys) are cleared by a bit a key, four words a row: with comparisons of
// every key's number, one to three of them, 2,048 tokens of 12 heads took 37.9 us, so 33.9, behind a window of 200 20.9 and 16.1, of 28 heads
// 39.4 and 28.3 (a window of 512 and four kept keys 44.4 and 34.4).
// A row's 128 scores stay in registers between the maximum and the exponentials (they were read twice), and the product with the
// values begins with the first 64 keys' probabilities: 162 -> 151.
// Blocks left over behind whole rounds of 148 would cost a round: they are cut into parts of their keys
// that prefill_merge_kernel adds up (192 -> 162; 512 tokens behind 3,000 of 12 heads, where 24 blocks are all there is, 62 -> 30).
//
// Keys outside a row's range get weight zero; what the cache holds there is finite (the pool
// starts as zeros and only finite values are written to it).  Page sizes: powers of two from
// 16; head sizes 64 and 128.  Every wait is bounded; a wait that runs out sets *error_flag.
#include "common.cuh"
#include "prefill_item.cuh"
#include "ptx_sm100.cuh"

namespace ifx {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ uint64_t desc_kmajor_sw128(uint32_t addr) {
  // rows of 128 bytes, 8-row groups 1024 bytes apart
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}
__device__ __forceinline__ uint64_t desc_mnmajor_sw128(uint32_t addr, uint32_t atom_stride_bytes) {
  // 64 MN elements (128 bytes) contiguous, the next 64 `atom_stride_bytes` further; K rows 128 bytes
  // apart, 8-row groups 1024 bytes apart
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((atom_stride_bytes >> 4) & 0x3FFF) << 16) |
         ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&r)[32]) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]),
        "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]),
        "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16f(uint32_t taddr, float (&r)[16]) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The largest of three.
__device__ __forceinline__ float max3(float x, float y, float z) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(x), "f"(y), "f"(z));
  return m;
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&u)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
      "%30,%31,%32};"
      ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]),
        "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(u[16]), "r"(u[17]),
        "r"(u[18]), "r"(u[19]), "r"(u[20]), "r"(u[21]), "r"(u[22]), "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]),
        "r"(u[27]), "r"(u[28]), "r"(u[29]), "r"(u[30]), "r"(u[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

constexpr int kSms = 148;                  // blocks of a round: one an SM
constexpr float kRescaleStep = 8.0f;      // log2 units the maximum may outgrow its reference before O is rescaled
constexpr uint32_t kTmemCols = 512;       // per query tile: scores (128 columns) and output (head size)
constexpr int kThreads = 384;             // fetch warp, MMA warp, two that rest, two softmax groups of four warps
constexpr int kNextSlots = 4;             // answers about the next block that are kept (see next_of)
// Registers a thread: the launch's 168 x 384 shared out anew, the softmax groups' 256 threads 208 and the others 88.
constexpr int kRegsSoftmax = 208, kRegsOther = 88;
static_assert(256 * kRegsSoftmax + 128 * kRegsOther <= 168 * kThreads, "no more than the block was launched with");

template <int D>
struct PrefillLayout {
  static constexpr int HALVES = D / 64;                       // 64-element (128-byte) column blocks of a head
  static constexpr int SLOTS = D == 128 ? 5 : 8;              // key or value tiles in flight
  static constexpr uint32_t Q_BYTES = HALVES * kBM * 128;     // one query tile: [half][128 rows][128 B]
  static constexpr uint32_t SLOT_BYTES = HALVES * kBN * 128;  // the keys or the values of one tile
  // barriers: queries there, their place free again, slots there and free, scores, probabilities of the first keys and of all,
  // output, the next block's number there and read by every role
  static constexpr int B_Q = 0, B_Q_FREE = B_Q + 2, B_FULL = B_Q_FREE + 2, B_EMPTY = B_FULL + SLOTS, B_S_FULL = B_EMPTY + SLOTS,
                       B_P_HALF = B_S_FULL + 2, B_P_FULL = B_P_HALF + 2, B_O_FULL = B_P_FULL + 2, B_NEXT = B_O_FULL + 2,
                       B_NEXT_FREE = B_NEXT + kNextSlots, B_COUNT = B_NEXT_FREE + kNextSlots;
  static constexpr size_t SMEM = 1024 + 2 * Q_BYTES + (size_t)SLOTS * SLOT_BYTES + kNextSlots * 16 + B_COUNT * 8 + 16;
};

// A block that has not begun is taken off the grid, and its number written to `answer` (16 bytes of shared memory).
__device__ __forceinline__ void take_next_block(uint32_t answer, uint32_t bar) {
  mbar_expect_tx(bar, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(answer), "r"(bar)
               : "memory");
}
// The number taken, -1 where every block had begun (or, with `ok` false, the answer never came).
__device__ __forceinline__ int next_block(uint32_t answer, uint32_t bar, uint32_t parity, bool& ok) {
  ok = __all_sync(0xffffffffu, mbar_wait(bar, parity));
  if (!ok) return -1;
  uint32_t there, x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 a;\n\t"
      "ld.shared.b128 a, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n\t"
      "selp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, a;\n\t}"
      : "=r"(there), "=r"(x)
      : "r"(answer)
      : "memory");
  fence_proxy_async_smem();
  return there ? (int)x : -1;
}

template <int D, bool KEPT>
__global__ void __launch_bounds__(kThreads, 1)
attn_prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap pool_map,
                            const int* __restrict__ block_table, const int* __restrict__ tiles,
                            const int* __restrict__ req_slot, bf16* __restrict__ out, int nq, int nkv, int page_size,
                            int page_shift, int max_blocks, int num_pages, KeyMask window, HeadOutput post, float scale_log2,
                            int* __restrict__ error_flag, int num_tiles, PrefillParts split) {
  using L = PrefillLayout<D>;
  using Item = PrefillItem<KEPT>;
  constexpr int HALVES = L::HALVES, SLOTS = L::SLOTS;
  constexpr uint32_t Q_BYTES = L::Q_BYTES, SLOT_BYTES = L::SLOT_BYTES;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  const uint32_t q_s = smem_addr(smem);                  // two query tiles
  const uint32_t kv_s = q_s + 2 * Q_BYTES;               // the ring of slots
  const uint32_t next_s = kv_s + SLOTS * SLOT_BYTES;     // answers about the next block
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * Q_BYTES + SLOTS * SLOT_BYTES + kNextSlots * 16);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + L::B_COUNT);
  const uint32_t bar0 = smem_addr(bars);
  auto bar = [&](int i) { return bar0 + 8 * i; };

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(bar(L::B_FULL + s), 1);
      mbar_init(bar(L::B_EMPTY + s), 1);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(bar(L::B_Q + q), 1);
      mbar_init(bar(L::B_Q_FREE + q), 4);
      mbar_init(bar(L::B_S_FULL + q), 1);
      mbar_init(bar(L::B_P_HALF + q), 4);
      mbar_init(bar(L::B_P_FULL + q), 4);
      mbar_init(bar(L::B_O_FULL + q), 1);
    }
    for (int s = 0; s < kNextSlots; ++s) {
      mbar_init(bar(L::B_NEXT + s), 1);
      mbar_init(bar(L::B_NEXT_FREE + s), 9);               // the MMA warp and the softmax groups' eight
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_holder)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_s = tmem_base, tmem_o = tmem_base + 2 * kBN;       // S of tile q: + q * 128; O: + q * D
  pdl_wait();

  // Every role goes through the same blocks: this one, then those that the fetching warp takes off the grid.  An answer's place is
  // free for the fourth one behind it when all others have read it: a softmax group without rows may be that far behind.
  auto next_of = [&](int n, bool& ok) {                    // the block behind the n-th
    return next_block(next_s + (n % kNextSlots) * 16, bar(L::B_NEXT + n % kNextSlots), (n / kNextSlots) & 1, ok);
  };
  auto next_read = [&](int n) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(L::B_NEXT_FREE + n % kNextSlots));
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    if (warp == 0) {
      // ---------------------------------------------------------------- fetching
      bool ok = true;
      int base = 0;                                         // slots used by the blocks before
      int loads[2] = {0, 0};                                // of query tile q
      int issued = 0;                                       // slots filled so far
      for (int n = 0, block = blockIdx.x; ok && block >= 0; ++n) {
        const Item it(block, tiles, num_tiles, nq, window, split);
        const int* table = block_table + (size_t)req_slot[it.r] * max_blocks;
        const int g = it.h / (nq / nkv);
        const int kfirst = window.first(it.pos0), kend = it.pos0 + it.rows;
        // the queries go over the output rows of the block before once those have left
        auto fetch_queries = [&]() {
          for (int q = 0; q < 2 && ok; ++q) {
            if (!it.has(q)) continue;
            if (loads[q] > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_Q_FREE + q), (loads[q] - 1) & 1));
            if (!ok) break;
            if (lane == 0) {
              mbar_expect_tx(bar(L::B_Q + q), Q_BYTES);
#pragma unroll
              for (int hh = 0; hh < HALVES; ++hh)
                tma_load_2d(q_s + q * Q_BYTES + hh * kBM * 128, &q_map, it.h * D + hh * 64, it.row0 + q * kBM, bar(L::B_Q + q));
            }
            ++loads[q];
          }
        };
        if (it.tb >= it.te) fetch_queries();               // (a part without keys)
        for (int kt = it.tb; kt < it.te && ok; kt = it.next_tile(kt)) {
          // lanes 0-7 take one 16-key block each; its page is looked up before the wait for a free slot
          const int key = kt * kBN + lane * 16;
          int page = 0, off = 0;
          // no visible key among the 16: any valid page, its keys get weight zero
          if (lane < kBN / 16 && key < kend && (key + 16 > kfirst || key < it.keep)) {
            page = table[key >> page_shift];
            if (page < 0 || page >= num_pages) page = 0;
            off = key & (page_size - 1);
          }
#pragma unroll 1
          for (int kv = 0; kv < 2 && ok; ++kv) {             // the keys, then the values
            if (kt == it.tb && kv == (n > 0 ? 1 : 0)) fetch_queries();     // (behind keys whose slot is free sooner)
            const int j = base + 2 * it.visited(kt) + kv, s = j % SLOTS;
            ok = ok && __all_sync(0xffffffffu, mbar_wait(bar(L::B_EMPTY + s), ((j / SLOTS) & 1) ^ 1));
            if (!ok) break;
            const uint32_t fb = bar(L::B_FULL + s);
            if (lane == 0) mbar_expect_tx(fb, SLOT_BYTES);
            __syncwarp();
            if (lane < kBN / 16) {
              const uint32_t dst = kv_s + s * SLOT_BYTES + lane * 2048;
              const int y = ((page * 2 + kv) * nkv + g) * page_size + off;
#pragma unroll
              for (int hh = 0; hh < HALVES; ++hh) tma_load_2d(dst + hh * kBN * 128, &pool_map, hh * 64, y, fb);
            }
            issued = j + 1;
          }
        }
        base += 2 * it.visits();
        // the next block is taken when this one's last tiles are on their way: late, so that SMs that are done sooner take more
        block = -1;
        if (ok && n >= kNextSlots) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_NEXT_FREE + n % kNextSlots), (n / kNextSlots - 1) & 1));
        if (ok) {
          if (lane == 0) take_next_block(next_s + (n % kNextSlots) * 16, bar(L::B_NEXT + n % kNextSlots));
          __syncwarp();
          block = next_of(n, ok);
        }
      }
      if (!ok && lane == 0) {
        atomicExch(error_flag, 7);
        for (int j = max(0, issued - SLOTS); j < issued; ++j)        // let the copies in flight land
          mbar_wait(bar(L::B_FULL + j % SLOTS), (j / SLOTS) & 1);
        for (int q = 0; q < 2; ++q)
          if (loads[q] > 0) mbar_wait(bar(L::B_Q + q), (loads[q] - 1) & 1);
      }
    } else if (warp == 1) {
      // ----------------------------------------------------- MMA issue: the warp in step, one lane's instructions by predicate
      const uint32_t elected = elect_one();
      const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kBN >> 3) << 17) |
                               ((uint32_t)(kBM >> 4) << 24);                       // both operands K-major
      const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(D >> 3) << 17) |
                               ((uint32_t)(kBM >> 4) << 24);                       // B (values) MN-major
      auto wait = [&](int b, int parity) { return (bool)__all_sync(0xffffffffu, mbar_wait(bar(b), parity)); };
      bool ok = true;
      int base = 0, loads[2] = {0, 0};
      int done[2] = {0, 0};                                // key tiles of each query tile so far
      for (int n = 0, block = blockIdx.x; ok && block >= 0; ++n) {
        const Item it(block, tiles, num_tiles, nq, window, split);
        auto last_q = [&](int kt) { return it.active(1, kt) ? 1 : 0; };    // the query tile that uses a key tile last
        auto issue_s = [&](int q, int kt) -> bool {         // S_q = Q_q . K(kt)^T
          const int j = base + 2 * it.visited(kt), s = j % SLOTS;
          if (!wait(L::B_FULL + s, (j / SLOTS) & 1)) return false;
          tc_fence_after();
          const uint32_t k_src = kv_s + s * SLOT_BYTES, q_src = q_s + q * Q_BYTES;
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t half = k / 4, inner = (k % 4) * 32;
            umma_ss(tmem_s + q * kBN, desc_kmajor_sw128(q_src + half * kBM * 128) + (inner >> 4),
                      desc_kmajor_sw128(k_src + half * kBN * 128) + (inner >> 4), idesc_s, k > 0 ? 1u : 0u, elected);
          }
          umma_commit(bar(L::B_S_FULL + q), elected);
          if (q == last_q(kt)) umma_commit(bar(L::B_EMPTY + s), elected);      // the keys have been read
          return true;
        };
        bool begun[2] = {false, false};
        auto issue_pv = [&](int q, int kt) -> bool {        // O_q += P_q . V(kt)
          const int j = base + 2 * it.visited(kt) + 1, s = j % SLOTS;
          if (!wait(L::B_FULL + s, (j / SLOTS) & 1)) return false;
          const uint32_t v_src = kv_s + s * SLOT_BYTES;
#pragma unroll
          for (int half = 0; half < 2; ++half) {             // the first 64 keys' probabilities are used while the others are made
            if (!wait((half ? L::B_P_FULL : L::B_P_HALF) + q, done[q] & 1)) return false;
            tc_fence_after();
#pragma unroll
            for (int k = half * (kBN / 32); k < (half + 1) * (kBN / 32); ++k)       // 16 keys (8 columns of pairs) a step
              umma_ts(tmem_o + q * D, tmem_s + q * kBN + k * 8, desc_mnmajor_sw128(v_src + k * 2048, kBN * 128),
                           idesc_o, (begun[q] || k > 0) ? 1u : 0u, elected);
          }
          umma_commit(bar(L::B_O_FULL + q), elected);
          if (q == last_q(kt)) umma_commit(bar(L::B_EMPTY + s), elected);      // the values have been read
          begun[q] = true;
          ++done[q];
          return true;
        };
        // The queries are waited for once a block, whether or not a part of it has keys for them.
        for (int q = 0; q < 2 && ok; ++q) {
          if (!it.has(q)) continue;
          ok = wait(L::B_Q + q, loads[q]++ & 1);
          if (ok && it.active(q, it.tb)) ok = issue_s(q, it.tb);
        }
        for (int kt = it.tb, before = it.tb; kt < it.te && ok; before = kt, kt = it.next_tile(kt)) {
          for (int q = 0; q < 2 && ok; ++q) {
            if (!it.active(q, kt)) continue;
            // a query tile that starts, or behind the kept keys goes on, later (window)
            if (kt != it.tb && (KEPT ? !it.active(q, before) : kt == (q == 0 ? it.tb_0 : it.tb_1))) ok = issue_s(q, kt);
            if (ok) ok = issue_pv(q, kt);
            // the next scores of this query tile go over its probabilities: the product that reads them
            // was issued just before and runs first; meanwhile the other tile's softmax is at work
            if (ok && it.active(q, it.next_tile(kt))) ok = issue_s(q, it.next_tile(kt));
          }
        }
        base += 2 * it.visits();
        block = -1;
        if (ok) {
          block = next_of(n, ok);
          next_read(n);
        }
      }
      if (!ok && lane == 0) atomicExch(error_flag, 8);
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------ softmax: one query tile, one row per thread
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    const int q = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                  // TMEM lane = query row of the tile
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_addr = tmem_s + q * kBN + lane_addr, o_addr = tmem_o + q * D + lane_addr;
    // where the warp's 32 rows of output lie before they leave: the place of its queries, which no product reads any more
    unsigned char* stage = smem + q * Q_BYTES + quarter * (32 * D * 2);
    constexpr int CHUNKS = D / 8;                          // of 16 bytes, in a row of 2 D bytes
    auto stage_at = [&](int r, int c) { return reinterpret_cast<uint4*>(stage + r * (D * 2) + ((c ^ (r & 7)) * 16)); };
    bool ok = true;
    int i0 = 0, loads = 0;                                // key tiles, and blocks with rows, of this query tile before this block
    for (int n = 0, block = blockIdx.x; ok && block >= 0; ++n) {
      const Item it(block, tiles, num_tiles, nq, window, split);
      const int rows_q = q == 0 ? min(it.rows, kBM) : it.rows_1;
      const int pos0_q = it.pos0 + q * kBM;
      const int pos = pos0_q + row;
      const int wfirst = window.first(pos);
      float m_ref = -INFINITY, l_run = 0.0f;
      int i = 0;                                            // key tiles of this query tile so far
      for (int kt = KEPT ? it.tb : (q == 0 ? it.tb_0 : it.tb_1); kt < (KEPT ? it.te : (q == 0 ? it.te_0 : it.te_1)); kt = it.next_tile(kt)) {
        if (KEPT && !it.active(q, kt)) continue;
        const int key0 = kt * kBN;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_S_FULL + q), (i0 + i) & 1));
        if (!ok) break;
        tc_fence_after();
        const bool edge = key0 + kBN - 1 > pos0_q ||
                          (window.any() && key0 < window.first(pos0_q + kBM - 1) && (!KEPT || key0 + kBN > it.keep));
        // the row's scores stay in registers: 128 of them
        float s[kBN];
#pragma unroll
        for (int c = 0; c < kBN; c += 32) tmem_ld32(s_addr + c, *reinterpret_cast<float(*)[32]>(&s[c]));
        tmem_wait_ld();
        if (edge) {                                          // a bit a key that the row sees: one test a score, whatever the mask
          auto below = [&](int end, int c) { return end <= c ? 0u : end >= c + 32 ? ~0u : (1u << (end - c)) - 1u; };
#pragma unroll
          for (int c = 0; c < kBN; c += 32) {
            const uint32_t sees = below(pos + 1 - key0, c) & (~below(wfirst - key0, c) | (KEPT ? below(it.keep - key0, c) : 0u));
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (!(sees >> j & 1)) s[c + j] = -INFINITY;
          }
        }
        float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int j = 4; j + 7 < kBN; j += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e) mx4[e] = max3(mx4[e], s[j + e], s[j + 4 + e]);
        const float mx = fmaxf(max3(mx4[0], mx4[1], max3(s[kBN - 4], s[kBN - 3], s[kBN - 2])), max3(mx4[2], mx4[3], s[kBN - 1]));
        // the reference maximum moves only when the row's maximum has outgrown it
        const bool outgrown = m_ref > -INFINITY && (mx - m_ref) * scale_log2 > kRescaleStep;
        float factor = 1.0f;
        if (outgrown) {
          factor = ex2((m_ref - mx) * scale_log2);
          m_ref = mx;
          l_run *= factor;
        } else if (m_ref == -INFINITY) {
          m_ref = mx;                                        // nothing accumulated for this row so far
        }
        if (i > 0 && __any_sync(0xffffffffu, outgrown)) {    // rescale this warp's rows of O in tensor memory
          ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_O_FULL + q), (i0 + i - 1) & 1));   // the products so far are done
          if (!ok) break;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            float t[32];
            tmem_ld32(o_addr + c, t);
            tmem_wait_ld();
            uint32_t u[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) u[j] = __float_as_uint(t[j] * factor);
            tmem_st32(o_addr + c, u);
          }
          tmem_wait_st();
        }
        // probabilities over the scores, 64 keys (32 columns of bfloat16 pairs) at a time; two scores an instruction
        const float bias = m_ref == -INFINITY ? 0.0f : -m_ref * scale_log2;
        const float2 scale2 = make_float2(scale_log2, scale_log2), bias2 = make_float2(bias, bias);
        float2 sum2[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
        for (int c = 0; c < kBN; c += 64) {
          uint32_t packed[32];
#pragma unroll
          for (int j = 0; j < 64; j += 4) {
            float pair[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float2 x = fma2(make_float2(s[c + j + 2 * e], s[c + j + 2 * e + 1]), scale2, bias2);
              const float2 p = make_float2(ex2(x.x), ex2(x.y));
              pair[e] = p.x + p.y;
              __nv_bfloat162 b2 = __floats2bfloat162_rn(p.x, p.y);
              packed[(j >> 1) + e] = *reinterpret_cast<uint32_t*>(&b2);
            }
            sum2[(j >> 2) & 1] = add2(sum2[(j >> 2) & 1], make_float2(pair[0], pair[1]));
          }
          tmem_st32(s_addr + (c >> 1), packed);              // columns whose scores have been read already
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar((c == 0 ? L::B_P_HALF : L::B_P_FULL) + q));
        }
        l_run += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
        ++i;
      }
      if (ok && i > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_O_FULL + q), (i0 + i - 1) & 1));
      if (ok && i == 0 && it.has(q)) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_Q + q), loads & 1));
      if (!ok) {
        if (lane == 0) atomicExch(error_flag, 9);
        break;
      }
      i0 += i;
      tc_fence_after();
      const int rows_w = rows_q - quarter * 32;             // rows of this warp
      if (!KEPT && it.slot >= 0) {                          // the sum as it is, for the merge
        const size_t at = (size_t)it.slot * 2 * kBM + q * kBM + quarter * 32;
        if (lane < rows_w)
          split.ml[at + lane] = i > 0 ? make_float2(m_ref > -INFINITY ? m_ref * scale_log2 : -INFINITY, l_run) : make_float2(-INFINITY, 0.0f);
        if (i > 0) {
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {            // rows of D / 2 float32 numbers
#pragma unroll
            for (int c = 0; c < D / 2; c += 32) {
              float t[32];
              tmem_ld32(o_addr + half * (D / 2) + c, t);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 32; j += 4)
                *stage_at(lane, (c + j) / 4) = make_uint4(__float_as_uint(t[j]), __float_as_uint(t[j + 1]), __float_as_uint(t[j + 2]),
                                                          __float_as_uint(t[j + 3]));
            }
            __syncwarp();
#pragma unroll 4
            for (int e = lane; e < 32 * CHUNKS; e += 32) {
              const int r = e / CHUNKS, c = e % CHUNKS;
              if (r < rows_w) *reinterpret_cast<uint4*>(split.o + (at + r) * D + half * (D / 2) + c * 4) = *stage_at(r, c);
            }
            __syncwarp();
          }
        }
      } else if (i > 0) {
        if (window.sink && m_ref > -INFINITY) l_run += exp2f(window.sink_log2(it.h) - m_ref * scale_log2);     // the sink's share
        const int t_row = it.row0 + q * kBM + min(row, max(rows_q - 1, 0));
        const float inv = (l_run > 0.0f ? 1.0f / l_run : 0.0f) * post.factor(t_row, it.h);
        if (post.table != nullptr) {                         // 16 pairs at a time: 32 columns, or 16 and their 16 partners
          const float4* cs4 = reinterpret_cast<const float4*>(post.table + (size_t)t_row * (D / 2));
          const int apart = post.interleaved ? 16 : D / 2;
#pragma unroll 1
          for (int m0 = 0; m0 < D / 2; m0 += 16) {
            const int c = post.interleaved ? 2 * m0 : m0;
            float lo[16], hi[16];
            tmem_ld16f(o_addr + c, lo);
            tmem_ld16f(o_addr + c + apart, hi);
            tmem_wait_ld();
            if (post.interleaved) {
#pragma unroll
              for (int j = 0; j < 8; j += 2) {
                const float4 a = cs4[(m0 + j) >> 1], b = cs4[(m0 + 8 + j) >> 1];
                HeadOutput::apply(make_float2(a.x, a.y), lo[2 * j], lo[2 * j + 1]);
                HeadOutput::apply(make_float2(a.z, a.w), lo[2 * j + 2], lo[2 * j + 3]);
                HeadOutput::apply(make_float2(b.x, b.y), hi[2 * j], hi[2 * j + 1]);
                HeadOutput::apply(make_float2(b.z, b.w), hi[2 * j + 2], hi[2 * j + 3]);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; j += 2) {
                const float4 a = cs4[(m0 + j) >> 1];
                HeadOutput::apply(make_float2(a.x, a.y), lo[j], hi[j]);
                HeadOutput::apply(make_float2(a.z, a.w), lo[j + 1], hi[j + 1]);
              }
            }
#pragma unroll
            for (int j = 0; j < 16; j += 8) {
              uint4 vl, vh;
              __nv_bfloat162* l2 = reinterpret_cast<__nv_bfloat162*>(&vl);
              __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&vh);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                l2[e] = __floats2bfloat162_rn(lo[j + 2 * e] * inv, lo[j + 2 * e + 1] * inv);
                h2[e] = __floats2bfloat162_rn(hi[j + 2 * e] * inv, hi[j + 2 * e + 1] * inv);
              }
              *stage_at(lane, (c + j) / 8) = vl;
              *stage_at(lane, (c + apart + j) / 8) = vh;
            }
          }
        } else {
#pragma unroll
          for (int c = 0; c < D; c += 32) {
            float t[32];
            tmem_ld32(o_addr + c, t);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint4 v;
              __nv_bfloat162* v2 = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
              for (int e = 0; e < 4; ++e) v2[e] = __floats2bfloat162_rn(t[j + 2 * e] * inv, t[j + 2 * e + 1] * inv);
              *stage_at(lane, (c + j) / 8) = v;
            }
          }
        }
        __syncwarp();
        bf16* dst = out + ((size_t)(it.row0 + q * kBM + quarter * 32) * nq + it.h) * D;
#pragma unroll 4
        for (int e = lane; e < 32 * CHUNKS; e += 32) {       // whole rows, 16 bytes a lane
          const int r = e / CHUNKS, c = e % CHUNKS;
          if (r < rows_w) *reinterpret_cast<uint4*>(dst + (size_t)r * nq * D + c * 8) = *stage_at(r, c);
        }
      }
      if (it.has(q)) {                                       // the next queries may come
        ++loads;
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(L::B_Q_FREE + q));
      }
      tc_fence_before();
      block = next_of(n, ok);
      next_read(n);
      if (!ok && lane == 0) atomicExch(error_flag, 9);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// grid (left over blocks, 32): a warp a row; parts in order.
template <int D>
__global__ void __launch_bounds__(256) prefill_merge_kernel(const int* __restrict__ tiles, bf16* __restrict__ out, int nq, int num_tiles,
                                                            PrefillParts split) {
  pdl_wait();
  const int block = split.full + blockIdx.x, row = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int* tile = tiles + (size_t)(num_tiles - 1 - block / nq) * 4;
  if (row >= tile[2]) return;
  const size_t at = (size_t)blockIdx.x * split.parts * 2 * kBM + row;
  // a lane a part's reference and sum (16 parts at most); then the parts' rows, four on their way at a time, added in order
  float2 mine = make_float2(-INFINITY, 0.0f);
  if (lane < split.parts) mine = split.ml[at + (size_t)lane * 2 * kBM];
  const float m = warp_max(mine.x);
  // a part without a key: its sums were not written (weight 0, and the row is not read)
  const bool there = lane < split.parts && !(mine.x == -INFINITY && !isnan(mine.y));
  const float w_mine = !there ? 0.0f : mine.x == -INFINITY ? 1.0f : exp2f(mine.x - m);
  const unsigned parts = __ballot_sync(0xffffffffu, there);
  float l = 0.0f;
  float acc[D / 32];
#pragma unroll
  for (int j = 0; j < D / 32; ++j) acc[j] = 0.0f;
  for (int p0 = 0; p0 < split.parts; p0 += 4) {
    float2 v[4][D / 64];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (parts >> (p0 + k) & 1) {
        const float* o = split.o + (at + (size_t)(p0 + k) * 2 * kBM) * D + lane * (D / 32);
#pragma unroll
        for (int j = 0; j < D / 64; ++j) v[k][j] = *reinterpret_cast<const float2*>(o + 2 * j);
      }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float w = __shfl_sync(0xffffffffu, w_mine, (p0 + k) & 31), sum = __shfl_sync(0xffffffffu, mine.y, (p0 + k) & 31);
      if (!(parts >> (p0 + k) & 1)) continue;
      l = fmaf(sum, w, l);
#pragma unroll
      for (int j = 0; j < D / 64; ++j) {
        acc[2 * j] = fmaf(v[k][j].x, w, acc[2 * j]);
        acc[2 * j + 1] = fmaf(v[k][j].y, w, acc[2 * j + 1]);
      }
    }
  }
  const float inv = l > 0.0f || isnan(l) ? 1.0f / l : 0.0f;
  bf16* to = out + ((size_t)(tile[1] + row) * nq + block % nq) * D + lane * (D / 32);
#pragma unroll
  for (int j = 0; j < D / 32; j += 2) *reinterpret_cast<__nv_bfloat162*>(to + j) = __floats2bfloat162_rn(acc[j] * inv, acc[j + 1] * inv);
}

template <int D, bool KEPT>
static int launch_prefill_tcgen05(const bf16* q, int num_tokens, const bf16* kv_pool, const int* block_table,
                                  const int* tiles, const int* req_slot, bf16* out, int num_tiles, int nq, int nkv,
                                  int page_size, int page_shift, int max_blocks, int num_pages, KeyMask window, HeadOutput post,
                                  float scale_log2, int* error_flag, cudaStream_t stream, int parts, void* workspace) {
  CUtensorMap q_map, pool_map;
  int rc = make_tensor_map_bf16(&q_map, q, num_tokens, nq * D, kBM);
  if (rc) return rc;
  rc = pool_tensor_map(&pool_map, kv_pool, (long long)num_pages * 2 * nkv * page_size, D);
  if (rc) return rc;
  const size_t smem = PrefillLayout<D>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_tcgen05_kernel<D, KEPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int blocks = nq * num_tiles, left = parts > 1 ? blocks % kSms : 0;
  PrefillParts split{parts == -1 ? 2 * blocks : blocks - left, parts, parts == -1, (float*)workspace, nullptr};
  if (left) split.ml = reinterpret_cast<float2*>(split.o + (size_t)left * parts * 2 * kBM * D);
  rc = launch_pdl(attn_prefill_tcgen05_kernel<D, KEPT>, dim3(split.full + left * parts), dim3(kThreads), smem, stream, 1, q_map,
                  pool_map, block_table, tiles, req_slot, out, nq, nkv, page_size, page_shift, max_blocks,
                  num_pages, window, post, scale_log2, error_flag, num_tiles, split);
  if (rc || !left) return rc;
  return launch_pdl(prefill_merge_kernel<D>, dim3(left, 2 * kBM / 8), dim3(256), 0, stream, 1, tiles, out, nq, num_tiles, split);
}

}  // namespace ifx

using namespace ifx;

extern "C" {

// 1 if the tensor-core kernel takes this head size and page size.
int ifx_attention_prefill_tcgen05_supports(int d, int page_size) {
  return (d == 64 || d == 128) && page_size >= 16 && (page_size & (page_size - 1)) == 0;
}

// q [num_tokens, nq * d] bfloat16, 16-byte aligned.  tiles: int32 [num_tiles, 4] = (request index, first
// flat row, rows <= 256, first position).
// chunk, sink, keep_first: see KeyMask; head_gate: null, or float32 [tokens, nq], see HeadOutput (common.cuh).
// sink_values: null, or one learned number per query head (float32 [nq]) that takes the place of the sink's score 0.
// turn_back: null, or float2 [tokens, d / 2], see HeadOutput.
int ifx_attention_prefill_tcgen05_sink(const void* q, int num_tokens, const void* kv_pool, const int* block_table,
                                       const int* tiles, const int* req_slot, void* out, int num_tiles, int nq, int nkv,
                                       int d, int page_size, int max_blocks, int num_pages, int window_size, int chunk,
                                       int sink, const float* sink_values, float scale, const float* turn_back,
                                   int turn_interleaved, int keep_first, const float* head_gate, int* error_flag,
                                       cudaStream_t stream) {
  const KeyMask window{window_size, chunk, sink, sink_values, keep_first};
  const HeadOutput post{reinterpret_cast<const float2*>(turn_back), turn_interleaved, head_gate, nq};
  if (num_tiles <= 0) return 0;
  if (!ifx_attention_prefill_tcgen05_supports(d, page_size) || nq <= 0 || nkv <= 0 || nq % nkv || max_blocks <= 0 ||
      num_tiles > 65535 || !(scale > 0.0f) || error_flag == nullptr)
    return IFX_E_BADARG;
  int ps = 0;
  while ((1 << ps) < page_size) ++ps;
  const float scale_log2 = scale * 1.4426950408889634f;
  auto run = [&](auto launch) {
    return launch((const bf16*)q, num_tokens, (const bf16*)kv_pool, block_table, tiles, req_slot, (bf16*)out, num_tiles, nq, nkv,
                  page_size, ps, max_blocks, num_pages, window, post, scale_log2, error_flag, stream, 1, nullptr);
  };
  if (d == 64) return keep_first > 0 ? run(launch_prefill_tcgen05<64, true>) : run(launch_prefill_tcgen05<64, false>);
  return keep_first > 0 ? run(launch_prefill_tcgen05<128, true>) : run(launch_prefill_tcgen05<128, false>);
}

int ifx_attention_prefill_tcgen05_ex(const void* q, int num_tokens, const void* kv_pool, const int* block_table,
                                     const int* tiles, const int* req_slot, void* out, int num_tiles, int nq, int nkv,
                                     int d, int page_size, int max_blocks, int num_pages, int window_size, int chunk,
                                     int sink, float scale, int* error_flag, cudaStream_t stream) {
  return ifx_attention_prefill_tcgen05_sink(q, num_tokens, kv_pool, block_table, tiles, req_slot, out, num_tiles, nq, nkv, d,
                                            page_size, max_blocks, num_pages, window_size, chunk, sink, nullptr, scale, nullptr, 0, 0, nullptr, error_flag,
                                            stream);
}

int ifx_attention_prefill_tcgen05(const void* q, int num_tokens, const void* kv_pool, const int* block_table,
                                  const int* tiles, const int* req_slot, void* out, int num_tiles, int nq, int nkv,
                                  int d, int page_size, int max_blocks, int num_pages, int window, float scale,
                                  int* error_flag, cudaStream_t stream) {
  return ifx_attention_prefill_tcgen05_ex(q, num_tokens, kv_pool, block_table, tiles, req_slot, out, num_tiles, nq, nkv, d,
                                          page_size, max_blocks, num_pages, window, 0, 0, scale, error_flag, stream);
}

// Bytes of workspace that cutting the left over blocks into `parts` (at least two) needs.
long long ifx_attention_prefill_tcgen05_parts_bytes(int num_tiles, int nq, int d, int parts) {
  return parts > 1 ? (long long)((long long)num_tiles * nq % kSms) * parts * 2 * kBM * (d + 2) * 4 : 0;
}

// The plain form with the blocks left over behind whole rounds cut into `parts` parts of their keys (1: none; two launches with more), or
// (-1) with a block for each 128 rows.
int ifx_attention_prefill_tcgen05_parts(const void* q, int num_tokens, const void* kv_pool, const int* block_table, const int* tiles,
                                        const int* req_slot, void* out, int num_tiles, int nq, int nkv, int d, int page_size,
                                        int max_blocks, int num_pages, int window, float scale, int parts, void* workspace,
                                        int* error_flag, cudaStream_t stream) {
  if (parts <= 1 && parts != -1)
    return ifx_attention_prefill_tcgen05(q, num_tokens, kv_pool, block_table, tiles, req_slot, out, num_tiles, nq, nkv, d, page_size,
                                         max_blocks, num_pages, window, scale, error_flag, stream);
  if (num_tiles <= 0) return 0;
  if (!ifx_attention_prefill_tcgen05_supports(d, page_size) || nq <= 0 || nkv <= 0 || nq % nkv || max_blocks <= 0 || num_tiles > 65535 ||
      !(scale > 0.0f) || error_flag == nullptr || parts > 16 || (parts > 1 && (workspace == nullptr || (uintptr_t)workspace % 16)))
    return IFX_E_BADARG;
  int ps = 0;
  while ((1 << ps) < page_size) ++ps;
  const KeyMask mask{window, 0, 0, nullptr, 0};
  const HeadOutput post{nullptr, 0, nullptr, nq};
  auto launch = d == 64 ? launch_prefill_tcgen05<64, false> : launch_prefill_tcgen05<128, false>;
  return launch((const bf16*)q, num_tokens, (const bf16*)kv_pool, block_table, tiles, req_slot, (bf16*)out, num_tiles, nq, nkv, page_size, ps,
                max_blocks, num_pages, mask, post, scale * 1.4426950408889634f, error_flag, stream, parts, workspace);
}

}  // extern "C"
