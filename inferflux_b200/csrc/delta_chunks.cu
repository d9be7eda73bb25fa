// The recurrence of delta_rule.cu over long spans, a stretch of 64 tokens at a time, for heads of 64 channels.
//
//   S_t = diag(w_t) S_(t-1) - e_t (u_t^T S_(t-1)) + k_t v_t^T        e_t = a_t u_t, u_t the unit key
//   o_t = S_t^T r_t
//
// What is erased, x_t = u_t^T S_(t-1), depends on the tokens before through x itself: with S_0 the state in front of the
// stretch and products of decays written G, over the tokens of the stretch as rows
//
//   X + M X = N V + U S_0          M[t, s] = u_t . (e_s G_(t-1) / G_s),  N[t, s] = u_t . (k_s G_(t-1) / G_s)      s < t
//   O = A V - B X + R S_0          A[t, s] = r_t . (k_s G_t / G_s),      B[t, s] = r_t . (e_s G_t / G_s)          s <= t
//   S = diag(G_64) S_0 + K^T V - E^T X                                   K, E: keys and e times G_64 / G_s
//
// a unit lower triangular system, solved for the columns of [N V | U] so that everything is linear in S_0.  Three kernels, and the norm:
//
//   delta_local   per stretch and head: outputs without S_0, the queries that meet S_0, the matrix that carries S_0 on, what is added
//   delta_carry   the states in front of every stretch, one small product a stretch, 8 value channels a block
//   chunk_reach   (chunk_scan.cu) adds what S_0 brings to the outputs
//   gated_heads_full  (pair_mixer.cu) norm and gate
//
// A decay lies between 0.545 and 1, so products over half a stretch and their reciprocals stay below 3e8: G_t / G_s is taken as
// a product on the one side and a reciprocal on the other, both counted from the middle of the stretch.  Products of operands in
// three bfloat16 parts: delta_local's on the 5th-generation tensor cores (parts_tcgen05.cuh), the carry's and reach's by mma.sync
// (chunk_scan.cuh).  The triangular system goes by blocks of 16 rows: a block is substituted, and what it changes in the rows behind
// it is a product.
//
// A stretch that holds a number that is not finite, or in which one comes up that a scan would not have formed, is walked token by
// token.  The order of the sums depends on where a span is cut into steps, so the float32 run keeps the scan.
//
// Bound: delta_local, one block of 16 warps an SM (200 KB of operands): operands are cut, multiplied and added up in phases that wait
// for one another, and the substitution is a chain of four blocks.  2,048 tokens of 24 heads: 165.6 us with products by mma.sync, two
// blocks of 8 warps an SM; 127.0 on tcgen05 (123.7 with six products of parts instead of eight).  On the way: the substitution of all
// 64 rows written out took 33,000 cycles (40 KB of code, the instruction cache), one by one in a loop 11,000, by blocks of 16 with
// products behind them 4,000.  delta_rule.cu's three kernels take 658 us there, these with the norm 193.
// Error against 64 bits (2-norm, 2,048 tokens), products by mma.sync and these: state 5.43e-7 and 5.43e-7, outputs 5.10e-7 and 5.09e-7.
// Scan and products by mma.sync: parameters where trained models have them 5.2e-7 and 4.6e-7, decays near one 1.76e-6 and 1.70e-6,
// random ones 0.95e-7 and 1.00e-7.
#include "parts_tcgen05.cuh"

namespace ifx {

constexpr int kDcThreads = 512, kDcD = 64, kDcP = kPitchV;
constexpr float kDcFloor = 0.6065306597126334f;            // exp(-1/2)

struct DeltaChunkArgs {
  const float* proj; int ld;                                // r, k, v, g, a in column blocks of heads * 64
  const float* w_raw; const float* w0; const float* a_bias;
  float* state; long long state_slot_stride; const int* req_slot; const int* cu_seqlens;
  float* out;                                               // [T, heads 64]
  int requests, min_span, heads;                            // shorter spans are left to delta_scan
  float *local, *reach;                                     // [stretches, heads, v, k], [T, heads 64]
  uint32_t* trans;                                          // [stretches, heads] matrices [k, k] as the carry's operands, see trans_word
  int* bad;                                                 // [stretches, heads]: whether the matrix holds a number that is not finite
};

// A stretch's matrix lies as delta_carry's lanes take it in: for 16 rows and 16 columns three parts (Split), of each four words a
// lane.  The order is that of FragA, which is that of a product's result: whoever makes 16 x 16 numbers of it stores what it holds.
constexpr int kTransWords = 3 * kDcD * kDcD / 2;
__device__ __forceinline__ size_t trans_word(int row_block, int column_block, int part, int lane) {
  return ((size_t)((row_block * 4 + column_block) * 3 + part) * 32 + lane) * 4;
}
// A number from its parts: their sum, or the first one alone if that is not finite.
__device__ __forceinline__ float from_parts(uint32_t hi, uint32_t mid, uint32_t lo, int upper) {
  auto part = [&](uint32_t w) { return __uint_as_float(upper ? w & 0xffff0000u : w << 16); };
  const float h = part(hi);
  return splits(h) ? h + (part(mid) + part(lo)) : h;
}

// Shared memory of delta_local, bytes from the first 1,024 boundary.  Tiles as in parts_tcgen05.cuh, rows of 64 numbers.
struct DeltaLayout {
  static constexpr int P = kPitchA, FLOATS = kChunk * P * 4;                // a float32 matrix of 64 x 64
  static constexpr uint32_t UR = 0, KE = UR + 3 * 128 * 128, V = KE + 3 * 128 * 128, B = V + 3 * 64 * 128, U32 = B + 3 * 64 * 128, R32 = U32 + FLOATS,
                            M = R32 + FLOATS, MP = M + FLOATS, MID = MP + 3 * 64 * 128, END = MID + 256, BYTES = END + 256;
  static constexpr uint32_t NA = UR, X = UR, W = M;        // in their places later, or before
  static_assert(MP % 1024 == 0, "a tile's place");
  static constexpr size_t SMEM = 1024 + BYTES + 4096;     // (48 rows of M from row 48 on are read up to row 95)
};
// The same rows as float32, for a stretch that is walked token by token.
struct DeltaWalkLayout {
  static constexpr int TILE = kChunk * kDcP;
  static constexpr int R = 0, U = TILE, K = 2 * TILE, E = 3 * TILE, V = 4 * TILE, W = 5 * TILE, FLOATS = W + kChunk * kPitchA;
  static_assert(FLOATS * 4 <= (int)DeltaLayout::BYTES, "room");
};
__device__ __forceinline__ float dc_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// With [U; R] the 64 tokens' unit keys and queries as rows one below the other, decays counted from the middle:
//
//   [U; R] [K; E]^T                 = [N M; A B], of which the triangles count            rows are lanes of tensor memory
//   [V . ]^T [N; A]^T               = (N V)^T | (A V)^T                                   value channels are lanes from here on
//   (1 + M) [X | U]                 by substitution, a thread a column, in float32
//   [X | U]^T B^T, [X | U]^T E, V^T K     what outputs, what is left to the state before, and what is added are short of or made of
//
// All 512 threads add up products (16 columns of a lane, or twice 16); the four warps whose lanes are the columns substitute, under V^T K.
__global__ void __launch_bounds__(kDcThreads, 1) delta_local_kernel(const DeltaChunkArgs a, int* error_flag) {
  using L = DeltaLayout;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint64_t bar_s[3];
  __shared__ uint32_t tmem_holder;
  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31, h = blockIdx.y, HD = a.heads * kDcD;
  int first, n;
  if (!chunk_of(a.cu_seqlens, a.requests, a.min_span, blockIdx.x, first, n)) return;
  const size_t item = (size_t)blockIdx.x * a.heads + h;
  unsigned char* smem = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  const uint32_t base = smem_addr(smem), bar = smem_addr(bar_s);
  float *u32 = reinterpret_cast<float*>(smem + L::U32), *r32 = reinterpret_cast<float*>(smem + L::R32), *w_s = reinterpret_cast<float*>(smem + L::W),
        *m_s = reinterpret_cast<float*>(smem + L::M), *x_s = reinterpret_cast<float*>(smem + L::X), *mid = reinterpret_cast<float*>(smem + L::MID),
        *end = reinterpret_cast<float*>(smem + L::END);
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 8, 1);
    mbar_init(bar + 16, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_before();

  // ---------------------------------------------------------- rows: queries, keys, values, how much is erased, unit keys, decays
  struct Rows { float4 r, k, v, e, u, w; };
  auto token = [&](int piece) { return piece * 32 + (tid >> 4); };         // sixteen neighbouring lanes a token, four channels each
  const int c = (tid & 15) * 4;
  auto fetch = [&](int piece, Rows& x) {                                   // true: a number that is not finite
    const int t = token(piece);
    x.r = x.k = x.v = x.e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    x.w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    if (t < n) {
      const float* row = a.proj + (size_t)(first + t) * a.ld + h * kDcD + c;
      x.r = *reinterpret_cast<const float4*>(row);
      x.k = *reinterpret_cast<const float4*>(row + HD);
      x.v = *reinterpret_cast<const float4*>(row + 2 * HD);
      x.e = *reinterpret_cast<const float4*>(row + 4 * HD);
      x.w = *reinterpret_cast<const float4*>(a.w_raw + (size_t)(first + t) * HD + h * kDcD + c);
    }
  };
  auto finish = [&](int piece, Rows& x) {
    if (token(piece) < n) {
      const float4 b = *reinterpret_cast<const float4*>(a.a_bias + h * kDcD + c), w0 = *reinterpret_cast<const float4*>(a.w0 + h * kDcD + c);
      x.e.x = dc_sigmoid(x.e.x + b.x); x.e.y = dc_sigmoid(x.e.y + b.y); x.e.z = dc_sigmoid(x.e.z + b.z); x.e.w = dc_sigmoid(x.e.w + b.w);
      x.w.x = expf(-kDcFloor * dc_sigmoid(x.w.x + w0.x)); x.w.y = expf(-kDcFloor * dc_sigmoid(x.w.y + w0.y));
      x.w.z = expf(-kDcFloor * dc_sigmoid(x.w.z + w0.z)); x.w.w = expf(-kDcFloor * dc_sigmoid(x.w.w + w0.w));
    }
    float ss = fmaf(x.k.x, x.k.x, fmaf(x.k.y, x.k.y, fmaf(x.k.z, x.k.z, x.k.w * x.k.w)));
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = 1.0f / sqrtf(ss + 1e-6f);
    x.u = make_float4(x.k.x * inv, x.k.y * inv, x.k.z * inv, x.k.w * inv);
    x.e.x *= x.u.x; x.e.y *= x.u.y; x.e.z *= x.u.z; x.e.w *= x.u.w;
    return !splits(x.r) || !splits(x.k) || !splits(x.v) || !splits(x.e) || !splits(x.w) || !isfinite(ss);
  };
  float* out = a.out + (size_t)first * HD + h * kDcD;
  float* reach = a.reach + (size_t)first * HD + h * kDcD;
  float* local = a.local + item * kDcD * kDcD;
  uint32_t* trans = a.trans + item * kTransWords;

  auto walk = [&]() {                                      // token by token: 64 columns of values, 64 of the unit matrix
    using W = DeltaWalkLayout;
    float* f = reinterpret_cast<float*>(smem);
    __syncthreads();                                       // (what lies there has been read)
#pragma unroll 1
    for (int piece = 0; piece < 2; ++piece) {
      Rows x;
      fetch(piece, x);
      finish(piece, x);
      const int t = token(piece);
      *reinterpret_cast<float4*>(f + W::R + t * kDcP + c) = x.r;
      *reinterpret_cast<float4*>(f + W::K + t * kDcP + c) = x.k;
      *reinterpret_cast<float4*>(f + W::V + t * kDcP + c) = x.v;
      *reinterpret_cast<float4*>(f + W::E + t * kDcP + c) = x.e;
      *reinterpret_cast<float4*>(f + W::U + t * kDcP + c) = x.u;
      *reinterpret_cast<float4*>(f + W::W + t * kPitchA + c) = x.w;
    }
    __syncthreads();
    if (tid < 2 * kDcD) {
      const bool unit = tid >= kDcD;
      const int j = tid & (kDcD - 1);
      float S[kDcD];                                       // in local memory: this path is for correctness
#pragma unroll 1
      for (int i = 0; i < kDcD; ++i) S[i] = unit && i == j ? 1.0f : 0.0f;
#pragma unroll 1
      for (int t = 0; t < n; ++t) {
        float x = 0.0f, kept = 0.0f, c1 = 0.0f, c2 = 0.0f;  // the output from the state in front of the token, as delta_scan_kernel takes it
        const float v = unit ? 0.0f : f[W::V + t * kDcP + j];
#pragma unroll 1
        for (int i = 0; i < kDcD; ++i) {
          const float r = f[W::R + t * kDcP + i];
          x = fmaf(f[W::U + t * kDcP + i], S[i], x);
          kept = fmaf(r * f[W::W + t * kPitchA + i], S[i], kept);
          c1 = fmaf(r, f[W::E + t * kDcP + i], c1);
          c2 = fmaf(r, f[W::K + t * kDcP + i], c2);
        }
#pragma unroll 1
        for (int i = 0; i < kDcD; ++i) {
          const float w = f[W::W + t * kPitchA + i] * S[i];
          S[i] = fmaf(-f[W::E + t * kDcP + i], x, unit ? w : fmaf(f[W::K + t * kDcP + i], v, w));
        }
        const float o = fmaf(-c1, x, unit ? kept : fmaf(c2, v, kept));
        (unit ? reach : out)[(size_t)t * HD + j] = o;
      }
#pragma unroll 1
      for (int i = 0; i < kDcD; ++i) {
        if (unit) {
          Split x;
          x.set(S[i], 0.0f);
          const size_t word = trans_word(i >> 4, j >> 4, 0, (i & 7) * 4 + ((j & 7) >> 1)) + (j & 1) * 2 + ((i >> 3) & 1);
          const uint32_t parts[3] = {x.hi, x.mid, x.lo};
          for (int p = 0; p < 3; ++p) reinterpret_cast<uint16_t*>(trans + word + p * 128)[(j >> 3) & 1] = (uint16_t)parts[p];
        } else {
          local[j * kDcD + i] = S[i];
        }
      }
    }
    if (tid == 0) a.bad[item] = 1;
  };

  bool ok = true;
  auto fast = [&]() -> bool {                              // false: to be walked
    uint32_t largest = 0;                                  // of what is made here to be cut
    auto note = [&](float x) { largest = max(largest, magnitude(x)); };
    {
      Rows x[2];
      bool bad = false;
#pragma unroll
      for (int i = 0; i < 2; ++i) fetch(i, x[i]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        bad = finish(i, x[i]) || bad;
        *reinterpret_cast<float4*>(w_s + token(i) * L::P + c) = x[i].w;
      }
      if (__syncthreads_or(bad)) return false;
      // decays from the middle: w_s then holds G_t / G_31 for t > 31, its reciprocal up to there
      if (tid < 2 * kDcD) {
        const int ch = tid & (kDcD - 1);
        Product p;
        if (tid < kDcD) {
          float w = w_s[31 * L::P + ch];
          w_s[31 * L::P + ch] = 1.0f;
#pragma unroll 8
          for (int t = 30; t >= 0; --t) {
            p.times(w);
            w = w_s[t * L::P + ch];
            w_s[t * L::P + ch] = p.value();
          }
          p.times(w);
          mid[ch] = p.value();                             // from the stretch's beginning to the middle
        } else {
#pragma unroll 8
          for (int t = 32; t < kChunk; ++t) {
            p.times(w_s[t * L::P + ch]);
            w_s[t * L::P + ch] = p.value();
          }
          end[ch] = p.value();
        }
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = token(i);
        const float4 p = *reinterpret_cast<const float4*>(w_s + t * L::P + c), q = make_float4(1.0f / p.x, 1.0f / p.y, 1.0f / p.z, 1.0f / p.w);
        const bool late = t > 31;
        const float4 f = late ? p : q, back = late ? q : p;
        const float4 b4 = *reinterpret_cast<const float4*>((t == 0 ? mid : w_s + (t - 1) * L::P) + c);
        const float4 before = t > 32 ? b4 : make_float4(1.0f / b4.x, 1.0f / b4.y, 1.0f / b4.z, 1.0f / b4.w);
        auto times = [&](float4& y, const float4& g) {
          y.x *= g.x; y.y *= g.y; y.z *= g.z; y.w *= g.w;
          largest = tc_largest(largest, y);
        };
        times(x[i].r, f);
        times(x[i].u, before);
        times(x[i].k, back);
        times(x[i].e, back);
        largest = tc_largest(largest, x[i].v);
        *reinterpret_cast<float4*>(u32 + t * L::P + c) = x[i].u;
        *reinterpret_cast<float4*>(r32 + t * L::P + c) = x[i].r;
        tc_put<128, 64>(smem + L::UR, t, c, x[i].u);
        tc_put<128, 64>(smem + L::UR, 64 + t, c, x[i].r);
        tc_put<128, 64>(smem + L::KE, t, c, x[i].k);
        tc_put<128, 64>(smem + L::KE, 64 + t, c, x[i].e);
        tc_put<64, 64>(smem + L::V, t, c, x[i].v);
      }
    }
    fence_proxy_async_smem();
    if (__syncthreads_or(largest >= kTcCut)) return false;
    tc_after();
    const uint32_t tmem = tmem_holder, lanes = (uint32_t)((warp & 3) * 32) << 16;
    const int row = (warp & 3) * 32 + lane, quarter = warp >> 2, q0 = quarter * 16;
    const bool lower = row >= kDcD;                        // of the 128 lanes: queries, or key channels
    const bool issuer = warp == 4;                         // (the first four substitute: issued by one of them, 4 us a layer more)
    const int own = row & (kDcD - 1);
    uint2 phase = make_uint2(0u, 0u);
    const uint64_t d_ur = tc_k_major(base + L::UR), d_ke = tc_k_major(base + L::KE), d_b = tc_k_major(base + L::B),
                   d_v = tc_mn_major(base + L::V, 64 * 128), d_keys = tc_mn_major(base + L::KE, 128 * 128);
    constexpr uint32_t kWide = 128 * 128, kNarrow = 64 * 128;                // a part of a tile of 128 or 64 rows
    auto ss = [&](int cols, int a_mn, int b_mn) {
      return [=](uint32_t d, uint64_t x, uint64_t y, uint32_t on, uint32_t elected) { umma_ss(d, x, y, tc_idesc(cols, a_mn, b_mn), on, elected); };
    };
    auto nothing = [] {};
    float made[32] = {};
    ok = tc_product<128, 4, 4, 64>(made, tmem, lanes + q0, bar, phase, issuer, [&](int p, int ks) { return d_ur + ((p * kWide + ks * 32) >> 4); },
                                   [&](int p, int ks) { return d_ke + ((p * kWide + ks * 32) >> 4); }, ss(128, 0, 0), false, nothing) && ok;
    tc_add_small<64>(made, tmem, lanes + q0);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const bool counts = lower ? q0 + i <= own : q0 + i < own;
      made[i] = counts ? made[i] : 0.0f;                   // N, A
      made[16 + i] = counts ? made[16 + i] : 0.0f;         // M, B
      note(made[i]);
      note(made[16 + i]);
    }
    auto put_row = [&](unsigned char* tile, uint32_t part, int at_row, const float* v) {      // 16 numbers of a row from column q0
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const Cut c0(v[8 * j], v[8 * j + 1]), c1(v[8 * j + 2], v[8 * j + 3]), c2(v[8 * j + 4], v[8 * j + 5]), c3(v[8 * j + 6], v[8 * j + 7]);
        unsigned char* to = tile + at_row * 128 + (((quarter * 2 + j) ^ (at_row & 7)) << 4);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(to + p * part) = make_uint4(c0.part[p], c1.part[p], c2.part[p], c3.part[p]);
      }
    };
    put_row(smem + L::NA, kWide, row, made);
    if (lower) {
      put_row(smem + L::B, kNarrow, own, made + 16);
    } else {
      put_row(smem + L::MP, kNarrow, own, made + 16);
      if (quarter == own >> 4) {
#pragma unroll
        for (int i = 0; i < 16; ++i)                       // what lies within 16 tokens in float32, by columns from the diagonal on
          if (q0 + i < own) m_s[(q0 + i) * L::P + own - (q0 + i) - 1] = made[16 + i];
      }
    }
    fence_proxy_async_smem();
    tc_before();
    if (__syncthreads_or(largest >= kTcCut || !ok)) return false;
#pragma unroll
    for (int i = 0; i < 32; ++i) made[i] = 0.0f;
    ok = tc_product<128, 4, 4, 64>(made, tmem, lanes + q0, bar, phase, issuer, [&](int p, int ks) { return d_v + ((p * kNarrow + ks * 2048) >> 4); },
                                   [&](int p, int ks) { return d_ur + ((p * kWide + ks * 32) >> 4); }, ss(128, 1, 0), false, nothing) && ok;
    tc_add_small<64>(made, tmem, lanes + q0);
    if (!lower) {
#pragma unroll
      for (int i = 0; i < 16; ++i) x_s[(q0 + i) * L::P + own] = made[i];
    }
    float o[16], kv[16] = {};
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] = made[16 + i];
    if (__syncthreads_or(!ok)) return false;
    constexpr uint32_t kAt = 96, kTake = kAt + 5 * 64;      // behind the parts of [X | U]^T; what solved tokens take off others
    bool taken = true;
    ok = tc_product<64, 4, 5>(kv, tmem + kAt, lanes + q0, bar, phase, issuer, [&](int p, int ks) { return d_v + ((p * kNarrow + ks * 2048) >> 4); },
                              [&](int p, int ks) { return d_keys + ((p * kWide + ks * 2048) >> 4); }, ss(64, 1, 1), false, [&] {
      if (tid >= 2 * kDcD) return;
      // Sixteen tokens at a time in float32; what they take off those behind them is a product with 48 rows of M (beyond the last token:
      // whatever lies there, for columns that nobody looks at), and the others move up.  (All in float32, one by one: 11,000 cycles, and
      // 33,000 written out, which does not fit the instruction cache.)
      float x[kChunk];
      const float* column = (lower ? u32 : x_s) + own;
      const float f = lower ? mid[own] : 1.0f;             // U, counted from the beginning
#pragma unroll
      for (int t = 0; t < kChunk; ++t) x[t] = column[t * L::P] * f;
      const uint64_t d_m = tc_k_major(base + L::MP);
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {
        const float* m = m_s + s * 16 * L::P;
#pragma unroll
        for (int q = 0; q < 15; ++q) {
#pragma unroll
          for (int j = 0; j < 15 - q; j += 4) {
            const float4 m4 = *reinterpret_cast<const float4*>(m + q * L::P + j);
            x[q + 1 + j] = fmaf(-m4.x, x[q], x[q + 1 + j]);
            if (q + 2 + j < 16) x[q + 2 + j] = fmaf(-m4.y, x[q], x[q + 2 + j]);
            if (q + 3 + j < 16) x[q + 3 + j] = fmaf(-m4.z, x[q], x[q + 3 + j]);
            if (q + 4 + j < 16) x[q + 4 + j] = fmaf(-m4.w, x[q], x[q + 4 + j]);
          }
        }
        uint32_t pairs[3][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          note(x[2 * i]);
          note(x[2 * i + 1]);
          const Cut cut(x[2 * i], x[2 * i + 1]);
#pragma unroll
          for (int p = 0; p < 3; ++p) pairs[p][i] = cut.part[p];
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) tc_st8(tmem + lanes + p * 32 + s * 8, pairs[p]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        if (s == 3) break;
        tc_before();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (warp == 0) {
          tc_after();
          const uint32_t elected = elect_one();
          constexpr int PX[8] = {0, 1, 2, 2, 0, 1, 1, 0}, PY[8] = {0, 2, 1, 0, 2, 1, 0, 1};
#pragma unroll
          for (int i = 0; i < 8; ++i)
            umma_ts(tmem + (i == 0 ? kTake : kTake + 48), tmem + PX[i] * 32 + s * 8,
                    d_m + ((PY[i] * kNarrow + (s + 1) * 2048 + s * 32) >> 4), tc_idesc(48, 0, 0), i > 1 ? 1u : 0u, elected);
          umma_commit(bar + 16, elected);
          __syncwarp();
        }
        taken = __all_sync(0xffffffffu, mbar_wait(bar + 16, s & 1)) && taken;
        tc_after();
#pragma unroll
        for (int j = 0; j < 48; j += 8) {
          float big[8], small[8];
          tc_ld8(tmem + lanes + kTake + j, big);
          tc_ld8(tmem + lanes + kTake + 48 + j, small);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i) x[j + i] = x[j + i + 16] - (big[i] + small[i]);
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }) && ok;
    ok = ok && taken;
    tc_add_small(kv, tmem + kAt, lanes + q0);
    if (__syncthreads_or(largest >= kTcCut || !ok)) return false;
    auto ts = [&](int b_mn) {
      return [=](uint32_t d, uint32_t x, uint64_t y, uint32_t on, uint32_t elected) { umma_ts(d, x, y, tc_idesc(64, 0, b_mn), on, elected); };
    };
    auto x_u = [&](int p, int ks) { return tmem + p * 32 + ks * 8; };
    float b[16] = {}, e[16] = {};
    ok = tc_product<64, 4, 5>(b, tmem + kAt, lanes + q0, bar, phase, issuer, x_u, [&](int p, int ks) { return d_b + ((p * kNarrow + ks * 32) >> 4); },
                              ts(0), false, nothing) && ok;
    tc_add_small(b, tmem + kAt, lanes + q0);
    __syncthreads();                                       // the accumulators are free again
    ok = tc_product<64, 4, 5>(e, tmem + kAt, lanes + q0, bar, phase, issuer, x_u,
                              [&](int p, int ks) { return d_keys + ((kNarrow + p * kWide + ks * 2048) >> 4); }, ts(1), false, [&] {
      const float f = mid[own];
      float* to = (lower ? reach : out) + (size_t)q0 * HD + own;
      const float* r = r32 + q0 * L::P + own;
#pragma unroll
      for (int i = 0; i < 16; ++i, to += HD)
        if (q0 + i < n) *to = lower ? fmaf(r[i * L::P], f, -b[i]) : o[i] - b[i];
    }) && ok;
    tc_add_small(e, tmem + kAt, lanes + q0);
    bool lost = false;
    if (!lower) {
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 f = *reinterpret_cast<const float4*>(end + q0 + i);
        *reinterpret_cast<float4*>(local + own * kDcD + q0 + i) =
            make_float4((kv[i] - e[i]) * f.x, (kv[i + 1] - e[i + 1]) * f.y, (kv[i + 2] - e[i + 2]) * f.z, (kv[i + 3] - e[i + 3]) * f.w);
      }
    } else {
      // numbers (row q0 + i, column own) of the matrix; words hold two columns eight apart, and two rows eight apart are neighbours: a lane
      // takes four pairs of rows of its column and the one eight away
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float f = end[q0 + i];
        e[i] = (q0 + i == own ? f * mid[own] : 0.0f) - f * e[i];
        lost = lost || !splits(e[i]);
      }
      const bool second = lane & 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // the first lane of a pair keeps rows 0 .. 3 and 8 .. 11, the second one the others
        const float give_lo = second ? e[i] : e[i + 4], give_hi = second ? e[i + 8] : e[i + 12];
        const float got_lo = __shfl_xor_sync(0xffffffffu, give_lo, 8), got_hi = __shfl_xor_sync(0xffffffffu, give_hi, 8);
        const int r = i + (second ? 4 : 0);
        Split lo, hi;
        lo.set(second ? got_lo : e[i], second ? e[i + 4] : got_lo);
        hi.set(second ? got_hi : e[i + 8], second ? e[i + 12] : got_hi);
        uint32_t* to = trans + trans_word(quarter, own >> 4, 0, r * 4 + ((own & 7) >> 1)) + (own & 1) * 2;
        *reinterpret_cast<uint2*>(to) = make_uint2(lo.hi, hi.hi);
        *reinterpret_cast<uint2*>(to + 128) = make_uint2(lo.mid, hi.mid);
        *reinterpret_cast<uint2*>(to + 256) = make_uint2(lo.lo, hi.lo);
      }
    }
    lost = __syncthreads_or(lost);
    if (tid == 0) a.bad[item] = lost;
    return true;
  };
  if (!fast()) {
    if (__syncthreads_or(!ok)) {
      if (tid == 0) atomicExch(error_flag, 83);
    } else {
      walk();
    }
  } else if (!ok && lane == 0) {
    atomicExch(error_flag, 83);
  }
  tc_before();
  __syncthreads();
  if (warp == 0) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_holder), "r"(512) : "memory");
  }
}

// grid (requests, heads, 8): 8 value channels of a head along a request's stretches, 16 key channels of them a warp.  The next
// stretch's matrix is on its way into registers, cut into parts by the block that made it, while this one's product runs; the
// state is cut by whoever makes it and handed on through shared memory, one barrier a stretch.
// Bound: that chain (shared memory, eight products, the sums, the cut).  32 stretches of 24 heads: 57 us with the matrix through shared
// memory and both operands cut by every warp that reads them, two barriers more; so 29.
constexpr int kCarryThreads = 128, kCarryV = 8;

__global__ void __launch_bounds__(kCarryThreads) delta_carry_kernel(const DeltaChunkArgs a) {
  __shared__ __align__(16) uint2 s_s[2][3][4][32];         // the state's parts: [part][16 key channels][lane], the order of FragB
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * kCarryV;
  const int chunks = chunks_of(a.cu_seqlens[r + 1] - a.cu_seqlens[r], a.min_span);
  if (chunks == 0) return;
  const size_t base = (size_t)chunks_before(a.cu_seqlens, a.min_span, r) * a.heads + h;
  float* st = a.state + (long long)a.req_slot[r] * a.state_slot_stride + (size_t)h * kDcD * kDcD;      // [k, v]
  // this thread's numbers of the state, a product's order: key channels k0 and k0 + 8, value channels vc and vc + 1
  const int lr = lane >> 2, k0 = warp * 16 + lr, vc = v0 + 2 * (lane & 3);
  float x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = st[(k0 + (i >> 1) * 8) * kDcD + vc + (i & 1)];
  auto hand_on = [&](int buf) {                            // true: a number that is not finite, which parts would lose
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      Split p;
      p.set(x[i], x[2 + i]);
      const int to = (2 * (lane & 3) + i) * 8 + lr;        // the word of the lane (value channel, lr / 2) for its odd or even key channel
      reinterpret_cast<uint32_t*>(s_s[buf][0][warp])[to] = p.hi;
      reinterpret_cast<uint32_t*>(s_s[buf][1][warp])[to] = p.mid;
      reinterpret_cast<uint32_t*>(s_s[buf][2][warp])[to] = p.lo;
    }
    return !splits(x[0]) || !splits(x[1]) || !splits(x[2]) || !splits(x[3]);
  };
  struct Next { uint4 m[4][3]; float l[4]; int bad; } ahead[3];           // two stretches on
  auto fetch = [&](Next& next, int c) {
    const size_t item = base + (size_t)min(c, chunks - 1) * a.heads;
    const uint32_t* m = a.trans + item * kTransWords;
    const float* l = a.local + item * kDcD * kDcD;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
      for (int p = 0; p < 3; ++p) next.m[kk][p] = *reinterpret_cast<const uint4*>(m + trans_word(warp, kk, p, lane));
#pragma unroll
    for (int i = 0; i < 4; ++i) next.l[i] = l[(vc + (i & 1)) * kDcD + k0 + (i >> 1) * 8];
    next.bad = a.bad[item];
  };
  fetch(ahead[0], 0);
  fetch(ahead[1], 1);
  bool bad = hand_on(0);
  auto step = [&](Next& now, Next& later, int c) {
    const size_t item = base + (size_t)c * a.heads;
    if (c + 2 < chunks) fetch(later, c + 2);               // (what is added to a stretch is read before its place takes a state)
#pragma unroll
    for (int i = 0; i < 4; ++i)                            // the state in front of the stretch
      a.local[item * kDcD * kDcD + (vc + (i & 1)) * kDcD + k0 + (i >> 1) * 8] = x[i];
    float acc[2][4] = {};
    const int buf = c & 1;
    const bool whole = !__syncthreads_or(bad) && !now.bad;
    if (!whole) {
#pragma unroll 1
      for (int j = 0; j < kDcD; ++j) {
        const uint32_t* m = a.trans + item * kTransWords + trans_word(warp, j >> 4, 0, lr * 4 + ((j & 7) >> 1)) + (j & 1) * 2;
        const int upper = (j >> 3) & 1;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int word = i >> 1;
          // (the state in front of the stretch, stored above: parts lose what lies below 2^-133)
          acc[0][i] = fmaf(from_parts(m[word], m[word + 128], m[word + 256], upper), a.local[item * kDcD * kDcD + (vc + (i & 1)) * kDcD + j], acc[0][i]);
        }
      }
    } else {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        FragA fa;
        FragB fb;
        const uint4 hi = now.m[kk][0], mid = now.m[kk][1], lo = now.m[kk][2];
        fa.v[0] = Split{hi.x, mid.x, lo.x};
        fa.v[1] = Split{hi.y, mid.y, lo.y};
        fa.v[2] = Split{hi.z, mid.z, lo.z};
        fa.v[3] = Split{hi.w, mid.w, lo.w};
        const uint2 shi = s_s[buf][0][kk][lane], smid = s_s[buf][1][kk][lane], slo = s_s[buf][2][kk][lane];
        fb.v[0] = Split{shi.x, smid.x, slo.x};
        fb.v[1] = Split{shi.y, smid.y, slo.y};
        mma_split(acc[kk & 1], fa, fb);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = acc[0][i] + acc[1][i] + now.l[i];
    bad = hand_on(buf ^ 1);
  };
  for (int c = 0; c < chunks; c += 3) {
    step(ahead[0], ahead[2], c);
    if (c + 1 < chunks) step(ahead[1], ahead[0], c + 1);
    if (c + 2 < chunks) step(ahead[2], ahead[1], c + 2);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) st[(k0 + (i >> 1) * 8) * kDcD + vc + (i & 1)] = x[i];
}

int launch_chunk_reach_64(const float* reach, const float* local, float* out, const int* cu_seqlens, int requests, int min_span, int heads,
                          int chunks, cudaStream_t stream);                                 // chunk_scan.cu
int launch_delta_scan(const float* proj, int ld, const float* w_raw, const float* w0, const float* a_bias, float* state,
                      long long slot_stride, const int* cu_seqlens, const int* req_slot, float* scratch, float* o, int num_requests, int T,
                      int heads, int dim, int max_span, cudaStream_t stream);               // delta_rule.cu
int launch_delta_finish(const float* o, const float* proj, int ld, const float* norm_w, float eps, void* y, int num_tokens, int heads,
                        int dim, int out_dtype, cudaStream_t stream);                       // delta_rule.cu

}  // namespace ifx

using namespace ifx;

extern "C" {

int ifx_delta_chunks_supports(int requests, int heads, int dim) {
  return requests > 0 && requests <= 64 && heads > 0 && heads <= 65535 && dim == kDcD;
}
long long ifx_delta_chunks_scratch_floats(int num_tokens, int requests, int min_span, int heads) {
  const long long items = (long long)chunks_at_most(num_tokens, requests, min_span) * heads;
  return items * (kDcD * kDcD + kTransWords) + (items + 3) / 4 * 4 + 2LL * num_tokens * heads * kDcD;
}

// As ifx_delta_rule_scan (delta_rule.cu) for heads of 64 channels, with scratch as above; rows on 16-byte boundaries.  Spans of
// fewer than min_span tokens go through delta_scan, with scan_scratch as ifx_delta_rule_scratch_floats says (null: there are none).
int ifx_delta_chunks_scan(const float* proj, int ld, const float* w_raw, const float* w0, const float* a_bias, const float* norm_w,
                          float eps, float* state, long long slot_stride, const int* cu_seqlens, const int* req_slot, float* scratch,
                          void* y, int num_requests, int num_tokens, int min_span, int heads, int dim, int out_dtype, float* scan_scratch,
                          int* error_flag, cudaStream_t stream) {
  if (num_tokens <= 0 || num_requests <= 0) return 0;
  if (!ifx_delta_chunks_supports(num_requests, heads, dim) || ld < 5 * heads * dim || slot_stride < (long long)heads * dim * dim ||
      scratch == nullptr || min_span < 1 || min_span > num_tokens)
    return IFX_E_BADARG;
  if (ld % 4 || ((uintptr_t)proj | (uintptr_t)w_raw | (uintptr_t)w0 | (uintptr_t)a_bias | (uintptr_t)scratch) % 16) return IFX_E_ALIGN;
  const int chunks = chunks_at_most(num_tokens, num_requests, min_span);
  DeltaChunkArgs a;
  a.proj = proj; a.ld = ld; a.w_raw = w_raw; a.w0 = w0; a.a_bias = a_bias;
  a.state = state; a.state_slot_stride = slot_stride; a.req_slot = req_slot; a.cu_seqlens = cu_seqlens;
  a.requests = num_requests; a.min_span = min_span; a.heads = heads;
  const size_t items = (size_t)chunks * heads, rows = (size_t)num_tokens * heads * kDcD;
  a.local = scratch;
  a.trans = reinterpret_cast<uint32_t*>(a.local + items * kDcD * kDcD);
  a.bad = reinterpret_cast<int*>(a.trans + items * kTransWords);
  a.reach = reinterpret_cast<float*>(a.bad + (items + 3) / 4 * 4);
  a.out = a.reach + rows;
  cudaError_t e = cudaFuncSetAttribute(delta_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DeltaLayout::SMEM);
  if (e != cudaSuccess) return (int)e;
  if (scan_scratch != nullptr) {
    const int rc = launch_delta_scan(proj, ld, w_raw, w0, a_bias, state, slot_stride, cu_seqlens, req_slot, scan_scratch, a.out, num_requests,
                                     num_tokens, heads, dim, min_span - 1, stream);
    if (rc) return rc;
  }
  delta_local_kernel<<<dim3(chunks, heads), kDcThreads, DeltaLayout::SMEM, stream>>>(a, error_flag);
  IFX_CHECK_LAUNCH();
  delta_carry_kernel<<<dim3(num_requests, heads, kDcD / kCarryV), kCarryThreads, 0, stream>>>(a);
  IFX_CHECK_LAUNCH();
  const int rc = launch_chunk_reach_64(a.reach, a.local, a.out, cu_seqlens, num_requests, min_span, heads, chunks, stream);
  if (rc) return rc;
  return launch_delta_finish(a.out, proj, ld, norm_w, eps, y, num_tokens, heads, dim, out_dtype, stream);
}

}  // extern "C"
