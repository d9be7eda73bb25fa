// Attention of decoded tokens over cached latents (bfloat16), latents of 256 numbers with 64 more rotated ones or none.
// What is computed is what latent_attention_mma.cu computes; that kernel, made for prompt tiles, gave a decoded token one warp
// that fetched, multiplied and waited in turn.  Here a block takes one token, up to 16 heads (the 16 rows of an
// mma.sync tile) and a stretch of keys; its four warps take turns at tiles of 16 keys, each on its own:
//
//   fetch    a tile is 16 cached rows of a page, boxes of [16 x 64] by TMA with the 128-byte swizzle; every warp has a ring of
//            two, asks for a tile as soon as it has read the one before last, and waits for nobody else
//   S, P, O  scores, running maximum and sum in float32, weights rounded to bfloat16 as the second product's operand, the
//            weighted sum of all 256 latent numbers in a warp's registers
//   end      the warps' sums meet in shared memory; with more than one stretch a token, latent_merge_kernel adds the stretches
//
// Two blocks an SM keep eight to sixteen tiles of 10 KB on their way.  Keys that a tile holds and the token does not see (behind
// its own position, in front of its window) are made zeros before they are read.  Waits are bounded and set *error_flag.
//
// Bound: HBM.  64 tokens of 12 heads at 1,600 to 16,000 keys (360 MB of latents): 457 -> 84 us (4.3 TB/s); 8 tokens of 28 heads at
// 400 to 4,000 keys 13 us, one token at 16,000 11 us.
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace ifx {

constexpr int kLdRank = 256, kLdWarps = 4, kLdStages = 2, kLdKeys = 16, kLdMaxStretch = 1024;

__device__ __forceinline__ void ld_ldsm(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ld_ldsm_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ld_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t ld_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// Byte offset of 8 numbers of a [16 rows][64 a box] tile as TMA's 128-byte swizzle leaves them; c8: number / 8.
__device__ __forceinline__ uint32_t ld_at(int row, int c8) { return (c8 >> 3) * 2048 + row * 128 + (((c8 & 7) ^ (row & 7)) << 4); }

template <int ROT>
struct LatentDecodeLayout {
  static constexpr int KW = kLdRank + ROT, BOXES = KW / 64;
  static constexpr uint32_t TILE = BOXES * 2048;
  static constexpr uint32_t Q = 0, RING = TILE, ROWS = RING + kLdWarps * kLdStages * TILE, BARS = ROWS + kLdMaxStretch / kLdKeys * 4,
                            ML = BARS + kLdWarps * kLdStages * 8, END = ML + kLdWarps * 16 * 8;
  static constexpr size_t BYTES = 1024 + END;
  static_assert(kLdWarps * 16 * kLdRank * 4 <= kLdWarps * kLdStages * TILE, "the warps' sums take the ring's place");
};

// grid (items of one token, groups of 16 heads, stretches)
template <int ROT>
__global__ void __launch_bounds__(kLdWarps * 32, 2) latent_decode_kernel(
    const __grid_constant__ CUtensorMap map, const __nv_bfloat16* __restrict__ ql, const int* __restrict__ block_table,
    const int4* __restrict__ items, const float* __restrict__ sinks, __nv_bfloat16* __restrict__ out, float* __restrict__ part_o,
    float2* __restrict__ part_ml, int total_rows, int heads, int page_size, int max_blocks, int num_pages, int window,
    float scale_log2, int stretch, const float* __restrict__ gate, int* __restrict__ error_flag) {
  using L = LatentDecodeLayout<ROT>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t base = smem_addr(smem);
  int* rows_s = reinterpret_cast<int*>(smem + L::ROWS);
  float2* ml_s = reinterpret_cast<float2*>(smem + L::ML);              // [warp][16]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int4 item = items[blockIdx.x];
  const int h0 = blockIdx.y * 16, nh = min(16, heads - h0);
  const int pos = item.w, hi = pos + 1, lo = window > 0 ? max(0, pos - window + 1) : 0;
  const int k0 = (lo & ~(kLdKeys - 1)) + blockIdx.z * stretch, k1 = min(hi, k0 + stretch);
  const size_t row0 = (size_t)item.y * heads + h0;                     // (token, head)
  if (k0 >= hi) {                                                      // this token's keys are fewer
    if (gridDim.z > 1 && tid < nh) part_ml[(size_t)blockIdx.z * total_rows + row0 + tid] = make_float2(-INFINITY, -1.0f);     // not written
    return;
  }
  const int tiles = (k1 - k0 + kLdKeys - 1) / kLdKeys;
  if (tid == 0) {
    for (int i = 0; i < kLdWarps * kLdStages; ++i) mbar_init(base + L::BARS + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < tiles; i += kLdWarps * 32) {                   // where every tile's rows lie in the pool
    const int key = k0 + i * kLdKeys;
    int page = block_table[(size_t)item.x * max_blocks + key / page_size];
    if (page < 0 || page >= num_pages) page = 0;                       // a broken table must not read outside the pool
    rows_s[i] = page * page_size + key % page_size;
  }
  __syncthreads();
  const uint32_t ring = base + L::RING + warp * kLdStages * L::TILE, bars = base + L::BARS + 8 * warp * kLdStages;
  auto fetch = [&](int tile, int slot) {                               // by one lane
    mbar_expect_tx(bars + 8 * slot, L::TILE);
#pragma unroll
    for (int b = 0; b < L::BOXES; ++b) tma_load_2d(ring + slot * L::TILE + b * 2048, &map, b * 64, rows_s[tile], bars + 8 * slot);
  };
  if (lane == 0)
    for (int s = 0; s < kLdStages; ++s)
      if (warp + s * kLdWarps < tiles) fetch(warp + s * kLdWarps, s);
  for (int i = tid; i < 16 * (L::KW / 8); i += kLdWarps * 32) {        // the heads' queries, zeros for rows without one
    const int r = i / (L::KW / 8), c8 = i % (L::KW / 8);
    const uint4 v = r < nh ? *reinterpret_cast<const uint4*>(ql + (row0 + r) * L::KW + c8 * 8) : make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(smem + L::Q + ld_at(r, c8)) = v;
  }
  __syncthreads();

  const int g = lane >> 2, quad = lane & 3, mi = lane >> 3, rr = lane & 7;
  float o[kLdRank / 8][4];
#pragma unroll
  for (int i = 0; i < kLdRank / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
  bool ok = true;
  int n = 0;                                                           // tiles of this warp so far
  for (int tile = warp; tile < tiles; tile += kLdWarps, ++n) {
    const int slot = n % kLdStages, key0 = k0 + tile * kLdKeys;
    ok = __all_sync(0xffffffffu, mbar_wait(bars + 8 * slot, (n / kLdStages) & 1));
    if (!ok) break;
    const uint32_t t_s = ring + slot * L::TILE;
    const bool edge = key0 < lo || key0 + kLdKeys > hi;
    if (edge) {                                                        // rows the token does not see become zeros
      for (int i = lane; i < kLdKeys * (L::KW / 8); i += 32) {
        const int r = i / (L::KW / 8);
        if (key0 + r < lo || key0 + r >= hi)
          *reinterpret_cast<uint4*>(smem + (t_s - base) + ld_at(r, i % (L::KW / 8))) = make_uint4(0u, 0u, 0u, 0u);
      }
      __syncwarp();
    }
    float s2[2][2][4] = {};                                            // [chain][8 keys]: two chains of products side by side
#pragma unroll
    for (int ks = 0; ks < L::KW / 16; ++ks) {
      uint32_t a[4], b[4];
      ld_ldsm(a, base + L::Q + ld_at(rr + (mi & 1) * 8, ks * 2 + (mi >> 1)));
      ld_ldsm(b, t_s + ld_at(rr + (mi >> 1) * 8, ks * 2 + (mi & 1)));
      ld_mma(s2[ks & 1][0], a, b[0], b[1]);
      ld_mma(s2[ks & 1][1], a, b[2], b[3]);
    }
    float s[2][4], m_new[2] = {m_run[0], m_run[1]};
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int key = key0 + j * 8 + quad * 2 + (c & 1);
        s[j][c] = (s2[0][j][c] + s2[1][j][c]) * scale_log2;
        if (edge && (key < lo || key >= hi)) s[j][c] = -INFINITY;
        m_new[c >> 1] = fmaxf(m_new[c >> 1], s[j][c]);
      }
    float corr[2], sum[2] = {0.0f, 0.0f};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      m_new[e] = fmaxf(m_new[e], __shfl_xor_sync(0xffffffffu, m_new[e], 1));
      m_new[e] = fmaxf(m_new[e], __shfl_xor_sync(0xffffffffu, m_new[e], 2));
      const float use = m_new[e] == -INFINITY ? 0.0f : m_new[e];
      corr[e] = exp2f(m_run[e] - use);                                 // exp2(-inf) = 0 at the start
      m_run[e] = m_new[e];
      m_new[e] = use;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s[j][c] = exp2f(s[j][c] - m_new[c >> 1]);
        sum[c >> 1] += s[j][c];
      }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 1);
      sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 2);
      l_run[e] = l_run[e] * corr[e] + sum[e];
    }
    if (__any_sync(0xffffffffu, corr[0] != 1.0f || corr[1] != 1.0f)) {
#pragma unroll
      for (int i = 0; i < kLdRank / 8; ++i) {
        o[i][0] *= corr[0]; o[i][1] *= corr[0]; o[i][2] *= corr[1]; o[i][3] *= corr[1];
      }
    }
    const uint32_t p[4] = {ld_pack(s[0][0], s[0][1]), ld_pack(s[0][2], s[0][3]), ld_pack(s[1][0], s[1][1]), ld_pack(s[1][2], s[1][3])};
#pragma unroll
    for (int c16 = 0; c16 < kLdRank / 16; ++c16) {
      uint32_t b[4];
      ld_ldsm_t(b, t_s + ld_at(rr + (mi & 1) * 8, c16 * 2 + (mi >> 1)));
      ld_mma(o[2 * c16], p, b[0], b[1]);
      ld_mma(o[2 * c16 + 1], p, b[2], b[3]);
    }
    fence_proxy_async_smem();                                          // this lane's reads and zeros, before the copy that goes over them
    __syncwarp();
    if (lane == 0 && tile + kLdStages * kLdWarps < tiles) fetch(tile + kLdStages * kLdWarps, slot);
  }
  if (!ok && lane == 0) {
    atomicExch(error_flag, 51);
    for (int s = 0; s < kLdStages; ++s) {                              // what may still be on its way
      const int i = n + s;
      if (warp + i * kLdWarps < tiles) mbar_wait(bars + 8 * (i % kLdStages), (i / kLdStages) & 1);
    }
  }
  if (quad == 0) {
    ml_s[warp * 16 + g] = make_float2(m_run[0], l_run[0]);
    ml_s[warp * 16 + g + 8] = make_float2(m_run[1], l_run[1]);
  }
  __syncthreads();                                                     // every warp is through with its ring
  float* sums = reinterpret_cast<float*>(smem + L::RING);              // [warp][16][256]
  float m_all[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
#pragma unroll
    for (int w = 0; w < kLdWarps; ++w) m_all[e] = fmaxf(m_all[e], ml_s[w * 16 + g + 8 * e].x);
    const float f = m_run[e] == -INFINITY ? 0.0f : exp2f(m_run[e] - m_all[e]);
    float* to = sums + (warp * 16 + g + 8 * e) * kLdRank + quad * 2;
#pragma unroll
    for (int i = 0; i < kLdRank / 8; ++i)                              // (pairs moved by the row's number: rows meet different banks)
      *reinterpret_cast<float2*>(to + (((i + g) & 31) * 8)) = make_float2(o[i][2 * e] * f, o[i][2 * e + 1] * f);
  }
  __syncthreads();
  for (int i = tid; i < nh * (kLdRank / 2); i += kLdWarps * 32) {
    const int r = i / (kLdRank / 2), c = (i % (kLdRank / 2)) * 2;
    const int at = ((((c >> 3) + (r & 7)) & 31) << 3) + (c & 7);
    float2 v = make_float2(0.0f, 0.0f);
    float m = -INFINITY, l = 0.0f;
#pragma unroll
    for (int w = 0; w < kLdWarps; ++w) {
      const float2 x = *reinterpret_cast<const float2*>(sums + (w * 16 + r) * kLdRank + at);
      v.x += x.x;
      v.y += x.y;
      m = fmaxf(m, ml_s[w * 16 + r].x);
    }
#pragma unroll
    for (int w = 0; w < kLdWarps; ++w)                                  // (0 times a sum that is not a number stays none)
      l = fmaf(ml_s[w * 16 + r].y, ml_s[w * 16 + r].x == -INFINITY ? 0.0f : exp2f(ml_s[w * 16 + r].x - m), l);
    if (gridDim.z > 1) {
      *reinterpret_cast<float2*>(part_o + ((size_t)blockIdx.z * total_rows + row0 + r) * kLdRank + c) = v;
      if (c == 0) part_ml[(size_t)blockIdx.z * total_rows + row0 + r] = make_float2(m, l);
    } else {
      float f = 1.0f;
      if (sinks != nullptr) {
        const float sk = sinks[h0 + r] * 1.4426950408889634f, mn = fmaxf(m, sk);
        f = exp2f(m - mn);
        l = l * f + exp2f(sk - mn);
      }
      const float inv = (l > 0.0f ? f / l : 0.0f) * (gate != nullptr ? gate[row0 + r] : 1.0f);
      *reinterpret_cast<uint32_t*>(out + (row0 + r) * kLdRank + c) = ld_pack(v.x * inv, v.y * inv);
    }
  }
}

int launch_latent_merge(const float* part_o, const float2* part_ml, const float* sinks, __nv_bfloat16* out, int total_rows, int heads,
                        int rank, int splits, const float* gate, cudaStream_t stream);       // latent_attention_mma.cu

}  // namespace ifx

using namespace ifx;

extern "C" {

int ifx_latent_decode_supports(int rank, int rot, int page_size) {
  return rank == kLdRank && (rot == 0 || rot == 64) && page_size > 0 && page_size % kLdKeys == 0;
}

// Keys of a stretch for a step of `tokens` decoded tokens that see up to `max_keys` each: four blocks for every SM to take turns
// at, a tile a warp at least, as many stretches as the merge takes at most.
int ifx_latent_decode_stretch(int tokens, int heads, int max_keys) {
  const long long blocks = (long long)tokens * ((heads + 15) / 16);
  long long stretch = ((long long)max_keys * blocks + 4 * 148 - 1) / (4 * 148);
  stretch = (stretch + 63) / 64 * 64;
  if (stretch < 64) stretch = 64;
  while (stretch < kLdMaxStretch && (max_keys + 15 + stretch - 1) / stretch > 64) stretch += 64;
  return stretch > kLdMaxStretch ? kLdMaxStretch : (int)stretch;
}

// As ifx_latent_attention_mma_rot (latent_attention_mma.cu) for items of one token; splits = stretches of `stretch` keys (a multiple
// of 64 up to 1,024) that cover max_keys + 15, at most 64; workspace as there.
int ifx_latent_decode(const void* ql, const void* pool, const int* block_table, const int* items, int num_items, const float* sinks,
                      void* out, void* workspace, int T, int heads, int rank, int rot, int page_size, int max_blocks, int num_pages,
                      int window, float scale, int stretch, int splits, const float* gate, int* error_flag, cudaStream_t stream) {
  if (num_items <= 0 || T <= 0) return 0;
  if (!ifx_latent_decode_supports(rank, rot, page_size) || heads <= 0 || max_blocks <= 0 || num_pages <= 0 || stretch <= 0 ||
      stretch % 64 || stretch > kLdMaxStretch || splits < 1 || splits > 64 || (heads + 15) / 16 > 65535 || error_flag == nullptr ||
      (splits > 1 && workspace == nullptr))
    return IFX_E_BADARG;
  if (((uintptr_t)ql | (uintptr_t)pool | (uintptr_t)out) % 16) return IFX_E_ALIGN;
  CUtensorMap map;
  int rc = pool_tensor_map(&map, pool, (long long)num_pages * page_size, rank + rot);
  if (rc) return rc;
  const int total_rows = T * heads;
  float* part_o = (float*)workspace;
  float2* part_ml = splits > 1 ? (float2*)(part_o + (size_t)splits * total_rows * rank) : nullptr;
  const dim3 grid(num_items, (heads + 15) / 16, splits);
  const float scale_log2 = scale * 1.4426950408889634f;
  auto run = [&](auto kern, size_t smem) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    kern<<<grid, kLdWarps * 32, smem, stream>>>(map, (const __nv_bfloat16*)ql, block_table, (const int4*)items, sinks, (__nv_bfloat16*)out,
                                                part_o, part_ml, total_rows, heads, page_size, max_blocks, num_pages, window, scale_log2,
                                                stretch, gate, error_flag);
    return (int)cudaGetLastError();
  };
  rc = rot ? run(latent_decode_kernel<64>, LatentDecodeLayout<64>::BYTES) : run(latent_decode_kernel<0>, LatentDecodeLayout<0>::BYTES);
  if (rc) return rc;
  return splits > 1 ? launch_latent_merge(part_o, part_ml, sinks, (__nv_bfloat16*)out, total_rows, heads, rank, splits, gate, stream) : 0;
}

}  // extern "C"
