// Attention of prompt portions over cached latents on the 5th-generation tensor cores (bfloat16), latents of 256 numbers with
// 64 more rotated ones or none.  What is computed is what latent_attention_mma.cu computes.
//
// A block takes 128 rows, neighbouring (token, head) pairs of one request, and walks the keys they see in tiles of 128.  A tile
// serves as keys (all its columns) and as values (the first 256):
//
//   S = Q . C^T     tcgen05.mma M 128 x N 128, inner size 256 + 64; two score buffers of 128 columns in tensor memory
//   P               two threads a row, 64 scores each in registers: running reference maximum (it moves when it has been
//                   outgrown by 2^8), exponentials, bfloat16 pairs over the scores
//   O += P . C      tcgen05.mma M 128 x N 256 with P from tensor memory; the tile as it lies is an MN-major operand
//
//   warp 0     TMA: the rows' queries once; per tile the pages' latents as boxes [16 keys x 64] into one of two buffers of 64 KB,
//              their rotated parts into one of 16 KB, which is free again as soon as the scores are made
//              (a buffer's first 64 keys leave when the first half of the weighted sum is done, and the next ones come in their place)
//   warp 1     MMA issue: the next tile's scores go in front of a tile's weighted sum, so that the exponentials of one tile run
//              under the products of the other; where the weights are there before the next tile's keys, the sum goes first,
//              since it frees the buffer that the tile behind that one waits for
//   warps 2-9  softmax: warps w and w + 4 share rows and meet once a tile for the maximum
//
// Shared memory is one block's (80 KB of queries, 144 KB of keys), tensor memory too (256 + 256 columns).
//
// Tiles of which not every row sees every key: cached numbers behind the block's last token are whatever a page's former owner
// left, and a token must not be touched by a key that only others of its block see.  The softmax warps clear the former, and
// rows of the latter kind that hold a number that is not finite, before the weighted sum reads them; a token that sees such a
// row has it in its scores.
//
// Every wait is bounded; a wait that runs out sets *error_flag.
//
// Bound: 2,304 cycles of the tensor pipe (576 multiply-adds a score) of the 3,830 that a tile takes, the rest the fetch of a tile,
// which begins only when one of the two buffers is free.  2,048 tokens of 12 heads (192 blocks on 148 SMs; one that holds the last
// tokens walks 16 tiles), us: latent_attention_mma_kernel and its merge 302; this with the scores always first, so that every sum
// waited for the next tile's fetch, 52.9 (3.2 a tile); whichever can go first 45.5 (2.3); fetched by halves, two scores an
// instruction and rows stored whole 44.4 (2.14).  1,000 tokens in three requests of 28 heads behind 1,500: 78.7, now 66.9; 300 of
// 12 heads behind 500 19.4 and 17.8.  Blocks of more than 12 tiles in two parts would save 5 and cost 3.5 for adding them up.
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace ifx {

constexpr int kLpRank = 256, kLpRows = 128, kLpKeys = 128, kLpThreads = 320;
constexpr float kLpRescaleStep = 8.0f;
constexpr uint32_t kLpBox = 128 * 128;                   // 128 rows of 64 numbers

__device__ __forceinline__ uint64_t lp_desc_k(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t lp_desc_mn(uint32_t addr) {          // the next 64 columns lie a box further
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(kLpBox >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void lp_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void lp_ld32(uint32_t taddr, float* r) {
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
__device__ __forceinline__ void lp_st32(uint32_t taddr, const uint32_t (&u)[32]) {
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
__device__ __forceinline__ void lp_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void lp_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void lp_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void lp_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float lp_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ bool lp_finite(uint32_t pair) {              // two bfloat16
  return (pair & 0x7f80u) != 0x7f80u && (pair & 0x7f800000u) != 0x7f800000u;
}

template <int ROT>
struct LatentPromptLayout {
  static constexpr int BOXES = (kLpRank + ROT) / 64, ROT_BOXES = ROT / 64;
  static constexpr uint32_t Q = 0, KV = Q + BOXES * kLpBox, KV_BYTES = 4 * kLpBox, TURNED = KV + 2 * KV_BYTES,
                            BARS = TURNED + ROT_BOXES * kLpBox;
  // B_KV_EMPTY: of a buffer's first 64 keys, + 2: of the others
  enum { B_Q = 0, B_KV_FULL = 1, B_KV_EMPTY = 3, B_ROT_FULL = 7, B_ROT_EMPTY = 8, B_S_FULL = 9, B_P_FULL = 11, B_O_FULL = 13, B_COUNT = 14 };
  static constexpr uint32_t HOLDER = BARS + B_COUNT * 8, MAXIMA = HOLDER + 8, END = MAXIMA + 2 * kLpRows * 4;
  static constexpr size_t BYTES = 1024 + END;
};

// grid (items x tiles of rows, 1, key parts).  items: (slot, first flat token, tokens <= 64, first position).
template <int ROT>
__global__ void __launch_bounds__(kLpThreads, 1) latent_prompt_kernel(
    const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap pool_map, const int* __restrict__ block_table,
    const int4* __restrict__ items, const float* __restrict__ sinks, __nv_bfloat16* __restrict__ out, float* __restrict__ part_o,
    float2* __restrict__ part_ml, int total_rows, int heads, int page_size, int max_blocks, int num_pages, int window,
    float scale_log2, int tiles_per_item, const float* __restrict__ gate, int* __restrict__ error_flag) {
  using L = LatentPromptLayout<ROT>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t base = smem_addr(smem), bars = base + L::BARS;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + L::HOLDER);
  float* maxima = reinterpret_cast<float*>(smem + L::MAXIMA);          // [half][128]
  __shared__ int odd_s;                                                // a cleared row held a number that is not finite
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int bx = gridDim.x - 1 - blockIdx.x;                           // later tokens see more keys: they start first
  const int4 item = items[bx / tiles_per_item];
  const int r0 = (bx % tiles_per_item) * kLpRows, rows_item = item.z * heads;
  if (r0 >= rows_item) return;
  const int rows = min(kLpRows, rows_item - r0);
  const int pos0 = item.w + r0 / heads, pos1 = item.w + (r0 + rows - 1) / heads;       // first and last token
  const size_t row0 = (size_t)item.y * heads + r0;
  const int first0 = window > 0 ? max(0, pos0 - window + 1) : 0, first1 = window > 0 ? max(0, pos1 - window + 1) : 0;   // their first keys
  int tb = first0 / kLpKeys, te = pos1 / kLpKeys + 1;
  if (gridDim.z > 1) {
    const int per = (te - tb + gridDim.z - 1) / gridDim.z;
    tb += blockIdx.z * per;
    te = min(te, tb + per);
    if (tb >= te) {
      if ((int)threadIdx.x < rows) part_ml[(size_t)blockIdx.z * total_rows + row0 + threadIdx.x] = make_float2(-INFINITY, -1.0f);   // not written
      return;
    }
  }
  const int n = te - tb;

  if (threadIdx.x == 0) {
    for (int i = 0; i < L::B_COUNT; ++i) mbar_init(bars + 8 * i, i == L::B_P_FULL || i == L::B_P_FULL + 1 ? 8 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    odd_s = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_holder)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  lp_before();
  __syncthreads();
  lp_after();
  const uint32_t tmem = *tmem_holder, tmem_o = tmem + 256;
  auto bar = [&](int i) { return bars + 8 * i; };

  if (warp == 0) {
    // ------------------------------------------------------------------ fetching
    const int* table = block_table + (size_t)item.x * max_blocks;
    if (lane == 0) {
      mbar_expect_tx(bar(L::B_Q), L::BOXES * kLpBox);
#pragma unroll
      for (int b = 0; b < L::BOXES; ++b) tma_load_2d(base + L::Q + b * kLpBox, &q_map, b * 64, (int)row0, bar(L::B_Q));
    }
    bool ok = true;
    int kv_issued = 0, rot_issued = 0;
    for (int i = 0; i < n && ok; ++i) {
      const int key = (tb + i) * kLpKeys + lane * 16;                  // lanes 0-7: 16 keys each
      int y = 0;
      if (lane < 8) {
        const int seen = min(max(key, first0 & ~15), pos1);            // outside what the rows see: a row they do, cleared later
        int page = table[seen / page_size];
        if (page < 0 || page >= num_pages) page = 0;
        y = page * page_size + (seen & ~15) % page_size;
      }
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {                           // 64 keys each, as the sums that read their places come to an end
        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_KV_EMPTY + 2 * part + (i & 1)), ((i >> 1) & 1) ^ 1));
        if (!ok && part == 0) break;                                   // (a tile that has begun is fetched whole, so that its copies land)
        if (part == 0 && lane == 0) mbar_expect_tx(bar(L::B_KV_FULL + (i & 1)), L::KV_BYTES);
        __syncwarp();
        if (lane >> 2 == part) {
          const uint32_t dst = base + L::KV + (i & 1) * L::KV_BYTES + lane * 2048;
#pragma unroll
          for (int b = 0; b < 4; ++b) tma_load_2d(dst + b * kLpBox, &pool_map, b * 64, y, bar(L::B_KV_FULL + (i & 1)));
        }
        kv_issued = i + 1;
      }
      if (!ok) break;
      if (ROT) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_ROT_EMPTY), (i & 1) ^ 1));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(bar(L::B_ROT_FULL), kLpBox);
        __syncwarp();
        if (lane < 8) tma_load_2d(base + L::TURNED + lane * 2048, &pool_map, kLpRank, y, bar(L::B_ROT_FULL));
        rot_issued = i + 1;
      }
    }
    if (!ok && lane == 0) {                                            // let the copies in flight land
      atomicExch(error_flag, 61);
      for (int i = max(0, kv_issued - 2); i < kv_issued; ++i) mbar_wait(bar(L::B_KV_FULL + (i & 1)), (i >> 1) & 1);
      if (rot_issued > 0) mbar_wait(bar(L::B_ROT_FULL), (rot_issued - 1) & 1);
      mbar_wait(bar(L::B_Q), 0);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------- MMA issue: the warp in step, one lane's instructions by predicate
    {
      const uint32_t elected = elect_one();
      auto wait = [&](int b, int parity) { return (bool)__all_sync(0xffffffffu, mbar_wait(bar(b), parity)); };
      auto ready = [&](int b, int parity) { return (bool)__all_sync(0xffffffffu, mbar_test(bar(b), parity)); };
      const uint32_t common = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kLpRows >> 4) << 24);
      const uint32_t idesc_s = common | ((uint32_t)(kLpKeys >> 3) << 17), idesc_o = common | (1u << 16) | ((uint32_t)(kLpRank >> 3) << 17);
      bool ok = wait(L::B_Q, 0);
      auto scores = [&](int i) -> bool {
        const uint32_t k_src = base + L::KV + (i & 1) * L::KV_BYTES, d = tmem + (i & 1) * kLpKeys;
        if (!wait(L::B_KV_FULL + (i & 1), (i >> 1) & 1)) return false;
        lp_after();
#pragma unroll
        for (int k = 0; k < kLpRank / 16; ++k)
          umma_ss(d, lp_desc_k(base + L::Q + (k / 4) * kLpBox) + (k % 4) * 2, lp_desc_k(k_src + (k / 4) * kLpBox) + (k % 4) * 2, idesc_s,
                    k > 0 ? 1u : 0u, elected);
        if (ROT) {
          if (!wait(L::B_ROT_FULL, i & 1)) return false;
          lp_after();
#pragma unroll
          for (int k = 0; k < ROT / 16; ++k)
            umma_ss(d, lp_desc_k(base + L::Q + 4 * kLpBox) + k * 2, lp_desc_k(base + L::TURNED) + k * 2, idesc_s, 1u, elected);
        }
        umma_commit(bar(L::B_S_FULL + (i & 1)), elected);
        if (ROT) umma_commit(bar(L::B_ROT_EMPTY), elected);
        return true;
      };
      if (ok) ok = scores(0);
      for (int i = 0; i < n && ok; ++i) {
        // whichever can go first: the next tile's scores (over the weights of tile i - 1, whose product was issued before) or this
        // tile's sum, which frees the buffer that the tile behind waits for
        bool made = i + 1 >= n;
        for (int tries = 0; !made && tries < kWaitLimit; ++tries) {
          if (ready(L::B_KV_FULL + ((i + 1) & 1), ((i + 1) >> 1) & 1)) {
            ok = scores(i + 1);
            made = true;
          } else if (ready(L::B_P_FULL + (i & 1), (i >> 1) & 1))
            break;
        }
        if (!ok || !(ok = wait(L::B_P_FULL + (i & 1), (i >> 1) & 1))) break;
        lp_after();
        const uint32_t v_src = base + L::KV + (i & 1) * L::KV_BYTES;
#pragma unroll
        for (int k = 0; k < kLpKeys / 16; ++k) {
          umma_ts(tmem_o, tmem + (i & 1) * kLpKeys + k * 8, lp_desc_mn(v_src + k * 2048), idesc_o, (i > 0 || k > 0) ? 1u : 0u, elected);
          if (k == kLpKeys / 32 - 1) umma_commit(bar(L::B_KV_EMPTY + (i & 1)), elected);
        }
        umma_commit(bar(L::B_KV_EMPTY + 2 + (i & 1)), elected);
        umma_commit(bar(L::B_O_FULL), elected);
        if (!made) ok = scores(i + 1);
      }
      if (!ok && lane == 0) atomicExch(error_flag, 62);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax: half the keys of a row a thread
    const int half = (warp - 2) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const int pos = item.w + (r0 + min(row, rows - 1)) / heads;
    const int first = window > 0 ? max(0, pos - window + 1) : 0;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    float m_ref = -INFINITY, l_run = 0.0f;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int key0 = (tb + i) * kLpKeys;
      const uint32_t s_addr = tmem + (i & 1) * kLpKeys + lane_addr;
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_S_FULL + (i & 1)), (i >> 1) & 1));   // (all go on to the barriers below)
      lp_after();
      float s[64];
      lp_ld32(s_addr + half * 64, s);
      lp_ld32(s_addr + half * 64 + 32, s + 32);
      lp_wait_ld();
      const bool edge = key0 + kLpKeys - 1 > pos0 || key0 < first1;    // not every row sees every key
      if (edge) {
        unsigned char* kv = smem + L::KV + (i & 1) * L::KV_BYTES;
        for (int r = warp - 2; r < kLpKeys; r += 8) {                  // a warp a row of 512 bytes
          const int key = key0 + r;
          if (key >= first1 && key <= pos0) continue;
          uint4* at = reinterpret_cast<uint4*>(kv + (lane >> 3) * kLpBox + r * 128 + (lane & 7) * 16);
          const uint4 v = *at;
          const bool odd = !(lp_finite(v.x) && lp_finite(v.y) && lp_finite(v.z) && lp_finite(v.w));
          const bool outside = key < first0 || key > pos1, clear = outside || __any_sync(0xffffffffu, odd);
          if (clear) *at = make_uint4(0u, 0u, 0u, 0u);
          if (clear && !outside && lane == 0) odd_s = 1;
        }
        fence_proxy_async_smem();
        asm volatile("bar.sync 6, 256;" ::: "memory");
        if (odd_s) {                                                   // a score that is not finite stays one whatever its weight
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (isinf(s[j])) s[j] = NAN;
        }
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const int key = key0 + half * 64 + j;
          if (key > pos || key < first) s[j] = -INFINITY;
        }
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 64; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], s[j]);
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      maxima[half * kLpRows + row] = mx;
      asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");   // with the warp of the row's other half
      mx = fmaxf(mx, maxima[(half ^ 1) * kLpRows + row]);
      const bool outgrown = m_ref > -INFINITY && (mx - m_ref) * scale_log2 > kLpRescaleStep;
      float factor = 1.0f;
      if (outgrown) {
        factor = lp_ex2((m_ref - mx) * scale_log2);
        m_ref = mx;
        l_run *= factor;
      } else if (m_ref == -INFINITY) {
        m_ref = mx;                                                    // nothing accumulated for this row so far
      }
      if (i > 0 && __any_sync(0xffffffffu, outgrown)) {                // this warp's half of its rows' sums in tensor memory
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_O_FULL), (i - 1) & 1));
        lp_after();
#pragma unroll 1
        for (int c = 0; c < 128; c += 32) {
          float t[32];
          uint32_t u[32];
          lp_ld32(tmem_o + lane_addr + half * 128 + c, t);
          lp_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) u[j] = __float_as_uint(t[j] * factor);
          lp_st32(tmem_o + lane_addr + half * 128 + c, u);
        }
      }
      const float bias = m_ref == -INFINITY ? 0.0f : -m_ref * scale_log2;
      const float2 scale2 = make_float2(scale_log2, scale_log2), bias2 = make_float2(bias, bias);
      float2 sum2[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
      uint32_t packed[32];
#pragma unroll
      for (int j = 0; j < 64; j += 4) {                                // two scores an instruction
        float2 p[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 x = fma2(make_float2(s[j + 2 * e], s[j + 2 * e + 1]), scale2, bias2);
          p[e] = make_float2(lp_ex2(x.x), lp_ex2(x.y));
          __nv_bfloat162 b2 = __floats2bfloat162_rn(p[e].x, p[e].y);
          packed[(j >> 1) + e] = *reinterpret_cast<uint32_t*>(&b2);
        }
        sum2[(j >> 2) & 1] = add2(sum2[(j >> 2) & 1], add2(make_float2(p[0].x, p[1].x), make_float2(p[0].y, p[1].y)));
      }
      lp_st32(s_addr + half * 32, packed);                             // columns whose scores both halves have read
      l_run += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
      lp_wait_st();
      lp_before();
      __syncwarp();
      if (lane == 0) lp_arrive(bar(L::B_P_FULL + (i & 1)));
      asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");   // the maxima are written again for the next tile
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::B_O_FULL), (n - 1) & 1));
    if (!ok && lane == 0) atomicExch(error_flag, 63);
    lp_after();
    maxima[half * kLpRows + row] = l_run;
    asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
    float l = l_run + maxima[(half ^ 1) * kLpRows + row];
    const size_t grow = row0 + min(row, rows - 1);
    if (gridDim.z > 1) {
      if (half == 0 && row < rows) part_ml[(size_t)blockIdx.z * total_rows + grow] = make_float2(m_ref > -INFINITY ? m_ref * scale_log2 : -INFINITY, l);
    } else if (sinks != nullptr && m_ref > -INFINITY) {
      l += exp2f(sinks[grow % heads] * 1.4426950408889634f - m_ref * scale_log2);
    }
    const float inv = (l > 0.0f || isnan(l) ? 1.0f / l : 0.0f) * (gate != nullptr ? gate[grow] : 1.0f);
    // Out through shared memory in whole rows of 256 bytes, where the queries lay: the products that read them are done.  (A
    // thread's own row, 16 bytes of 32 rows a store, took 2 us.)
    unsigned char* stage = smem + L::Q + (warp - 2) * (32 * 256);
    auto stage_at = [&](int r, int c) { return reinterpret_cast<uint4*>(stage + r * 256 + ((c ^ (r & 7)) * 16)); };
    const int rows_w = rows - quarter * 32;                            // rows of this warp
    if (gridDim.z > 1) {
#pragma unroll 1
      for (int c0 = half * 128; c0 < half * 128 + 128; c0 += 64) {
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          float t[32];
          lp_ld32(tmem_o + lane_addr + c0 + c, t);
          lp_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(stage_at(lane, (c + j) / 4)) = make_float4(t[j], t[j + 1], t[j + 2], t[j + 3]);
        }
        __syncwarp();
        float* to = part_o + ((size_t)blockIdx.z * total_rows + row0 + quarter * 32) * kLpRank + c0;
#pragma unroll 4
        for (int e = lane; e < 32 * 16; e += 32)
          if ((e >> 4) < rows_w) *reinterpret_cast<uint4*>(to + (size_t)(e >> 4) * kLpRank + (e & 15) * 4) = *stage_at(e >> 4, e & 15);
        __syncwarp();
      }
    } else {
#pragma unroll
      for (int c = 0; c < 128; c += 32) {
        float t[32];
        lp_ld32(tmem_o + lane_addr + half * 128 + c, t);
        lp_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          uint4 v;
          __nv_bfloat162* v2 = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
          for (int e = 0; e < 4; ++e) v2[e] = __floats2bfloat162_rn(t[j + 2 * e] * inv, t[j + 2 * e + 1] * inv);
          *stage_at(lane, (c + j) / 8) = v;
        }
      }
      __syncwarp();
      __nv_bfloat16* to = out + (row0 + quarter * 32) * kLpRank + half * 128;
#pragma unroll 4
      for (int e = lane; e < 32 * 16; e += 32)
        if ((e >> 4) < rows_w) *reinterpret_cast<uint4*>(to + (size_t)(e >> 4) * kLpRank + (e & 15) * 8) = *stage_at(e >> 4, e & 15);
    }
  }
  lp_before();
  __syncthreads();
  if (warp == 1) {
    lp_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

int launch_latent_merge(const float* part_o, const float2* part_ml, const float* sinks, __nv_bfloat16* out, int total_rows, int heads,
                        int rank, int splits, const float* gate, cudaStream_t stream);       // latent_attention_mma.cu

}  // namespace ifx

using namespace ifx;

extern "C" {

int ifx_latent_prompt_supports(int rank, int rot, int page_size) {
  return rank == kLpRank && (rot == 0 || rot == 64) && page_size > 0 && page_size % 16 == 0;
}

// As ifx_latent_attention_mma_rot (latent_attention_mma.cu): items of up to 64 tokens, workspace and splits as there (at most 16).
int ifx_latent_prompt(const void* ql, const void* pool, const int* block_table, const int* items, int num_items, int max_item_tokens,
                      const float* sinks, void* out, void* workspace, int T, int heads, int rank, int rot, int page_size, int max_blocks,
                      int num_pages, int window, float scale, int splits, const float* gate, int* error_flag, cudaStream_t stream) {
  if (num_items <= 0 || T <= 0) return 0;
  if (!ifx_latent_prompt_supports(rank, rot, page_size) || heads <= 0 || max_blocks <= 0 || num_pages <= 0 || max_item_tokens < 1 ||
      max_item_tokens > 64 || splits < 1 || splits > 16 || !(scale > 0.0f) || error_flag == nullptr || (splits > 1 && workspace == nullptr))
    return IFX_E_BADARG;
  if (((uintptr_t)ql | (uintptr_t)pool | (uintptr_t)out | (uintptr_t)workspace) % 16) return IFX_E_ALIGN;
  const long long tiles = ((long long)max_item_tokens * heads + kLpRows - 1) / kLpRows;
  if (tiles * num_items > 0x7fffffffLL || (long long)T * heads > 0x7fffffffLL) return IFX_E_TOOBIG;
  CUtensorMap q_map, pool_map;
  int rc = make_tensor_map_bf16(&q_map, ql, (long long)T * heads, rank + rot, kLpRows);
  if (rc) return rc;
  rc = pool_tensor_map(&pool_map, pool, (long long)num_pages * page_size, rank + rot);
  if (rc) return rc;
  const int total_rows = T * heads;
  float* part_o = (float*)workspace;
  float2* part_ml = splits > 1 ? (float2*)(part_o + (size_t)splits * total_rows * rank) : nullptr;
  const float scale_log2 = scale * 1.4426950408889634f;
  auto run = [&](auto kern, size_t smem) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    kern<<<dim3((unsigned)(tiles * num_items), 1, splits), kLpThreads, smem, stream>>>(
        q_map, pool_map, block_table, (const int4*)items, sinks, (__nv_bfloat16*)out, part_o, part_ml, total_rows, heads, page_size, max_blocks,
        num_pages, window, scale_log2, (int)tiles, gate, error_flag);
    return (int)cudaGetLastError();
  };
  rc = rot ? run(latent_prompt_kernel<64>, LatentPromptLayout<64>::BYTES) : run(latent_prompt_kernel<0>, LatentPromptLayout<0>::BYTES);
  if (rc) return rc;
  return splits > 1 ? launch_latent_merge(part_o, part_ml, sinks, (__nv_bfloat16*)out, total_rows, heads, rank, splits, gate, stream) : 0;
}

}  // extern "C"
