// The scans of chunk_scan.cu with one decay per head (constant, or from a step), a stretch of 128 tokens at a time on the
// 5th-generation tensor cores.  With S_0 the state in front of a stretch and d(t, s) the decays from s + 1 to t:
//
//   chunk_add      per stretch and head: sum over s of (k_s d(128, s)) v_s^T, and d over the whole stretch
//   chunk_carry    (chunk_scan.cu) the states in front of every stretch
//   chunk_outputs  o_t = d(t, begin) q_t^T S_0  +  sum over s <= t of (q_t . k_s) d(t, s) v_s
//
// Products of float32 operands in parts: parts_tcgen05.cuh.  Scores times decays go back as parts, to shared or to tensor memory.
//
// Decays: powers of the one number in float64; or, from steps, exp of differences of float64 sums.  Neither divides by a decay.
//
// A stretch that holds a number that cannot be cut, or makes one, is walked token by token from the state in front of it.
// Every wait is bounded; a wait that runs out sets *error_flag and the block's outputs are not written.
//
// Bound: chunk_outputs (one block an SM, 192 KB of operands) by phases that wait for one another: of 40,000 cycles a block of 128 x 128, reads
// and cuts of queries and keys 5,000, three products 5,600 to 7,000 each (3,100 of them the tensor pipe's), the state's and values' cuts
// 4,600 and 5,200, stores 5,800; all blocks meet each phase together, so memory is idle during products.  12 heads, 1,901 tokens of two
// requests: chunk_local 74.6, carry 11.5, reach 30.9 us -> 16.4, 8.0 and 43.9.
#include "parts_tcgen05.cuh"

namespace ifx {

constexpr int kTc = 128;                                   // tokens of a stretch

// -------------------------------------------------------------------------------------------- decays
// What a block knows of its tokens' decays: d(t, s) for s <= t, t = -1 the stretch's beginning for s (d(t, -1) takes in token 0).
template <int MODE>
struct TcDecay {
  float2 sum[kTc + 1];                                     // from steps: minus the logarithms up to token t - 1, as two numbers
  float power[kTc + 1];                                    // constant: powers
  float step[kTc];
  float key[kTc];                                          // from steps: the largest key number of a token (chunk_outputs)
  float rest[kTc];                                         // from steps: the decays behind a token to the end of its 16 tokens, times its step
  double warp_sum[4];

  // By all threads; barriers at its end.  True: a number that is not finite.
  __device__ __forceinline__ bool make(const ChunkArgs& a, int h, int first, int n) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    bool bad = false;
    double x = 0.0;
    if (MODE == CHUNK_STEP) {
      if (t < kTc) {
        float st = 0.0f;
        if (t < n) {
          st = chunk_softplus(a.raw[(size_t)(first + t) * a.raw_stride + h] + a.step_bias[h]);
          x = (double)expf(a.log_rate[h]) * (double)st;
        }
        step[t] = st;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
      }
      __syncthreads();
      if (t < kTc) {
        for (int w = 0; w < warp; ++w) x += warp_sum[w];
        const float hi = (float)x;
        sum[t + 1] = make_float2(hi, (float)(x - (double)hi));
        if (t == 0) sum[0] = make_float2(0.0f, 0.0f);
        bad = !(x < 3e38);
      }
    } else {
      if (t < kTc) {                                       // thread t: the power t + 1, its exponent's bits from the top
        const double w = a.rate[h];
        x = 1.0;
        for (int b = 7; b >= 0; --b) {
          x *= x;
          if ((t + 1) >> b & 1) x *= w;
        }
        power[t + 1] = (float)x;
        if (t == 0) power[0] = 1.0f;
        bad = !splits((float)x);
      }
      __syncthreads();
    }
    __syncthreads();
    if (MODE == CHUNK_STEP) {
      if (t < kTc) rest[t] = between(t + 1, (t | 15) + 1) * step[t];
      __syncthreads();
    }
    return bad;
  }
  // The decays of the tokens i .. j - 1.
  __device__ __forceinline__ float between(int i, int j) const {
    if (MODE != CHUNK_STEP) return power[j - i];
    const float2 a = sum[j], b = sum[i];
    const float d = a.x - b.x, bb = d - a.x, rest = ((a.x - (d - bb)) - (b.x + bb)) + (a.y - b.y);      // their difference as two numbers
    const float e = expf(-d);
    return fmaf(-rest, e, e);
  }
};

// -------------------------------------------------------------------------------------------- what a stretch adds
// The tokens come in two halves of 64 rows, so that two blocks share an SM.
template <int DK, int DV>
struct TcAdd {
  static constexpr int THREADS = 256, NX = 128, NY = DK == 128 ? DV : DK;      // rows and columns of the product: (k, v), or (v, k) for keys of 64
  static constexpr uint32_t X = 3 * 2 * 64 * 128, Y = 3 * (NY / 64) * 64 * 128;
  static constexpr size_t SMEM = 1024 + X + Y;
  static constexpr int COLUMNS = 256, SLOTS = COLUMNS / NY;
};

template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(256, 2) chunk_add_kernel(const ChunkArgs a, int* error_flag) {
  using L = TcAdd<DK, DV>;
  constexpr int NY = L::NY;
  extern __shared__ unsigned char smem_raw[];
  __shared__ TcDecay<MODE> decay;
  __shared__ uint64_t bar_s[2];
  __shared__ uint32_t tmem_holder;
  const int h = blockIdx.y, g = h / (a.heads / a.groups);
  int first, n;
  if (!chunk_of(a.cu_seqlens, a.requests, a.min_span, blockIdx.x, first, n, kTc)) return;
  const size_t item = (size_t)blockIdx.x * a.heads + h;
  unsigned char* smem = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  const uint32_t x0 = smem_addr(smem), y0 = x0 + L::X, bar = smem_addr(bar_s);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)), "r"((uint32_t)L::COLUMNS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_before();
  bool bad = decay.make(a, h, first, n);                   // (its barriers are the allocation's, too)
  tc_after();
  const uint32_t tmem = tmem_holder;

  if (threadIdx.x == 0) {                                  // the whole stretch's decay as two numbers
    double d;
    if (MODE == CHUNK_STEP) {
      d = exp(-((double)decay.sum[n].x + (double)decay.sum[n].y));
    } else {
      d = 1.0;
      for (int b = 7; b >= 0; --b) {
        d *= d;
        if (n >> b & 1) d *= (double)a.rate[h];
      }
    }
    const float hi = (float)d;
    a.total[2 * item] = hi;
    a.total[2 * item + 1] = (float)(d - (double)hi);
  }

  bool ok = true;
  uint32_t largest = 0;
  uint2 phase = make_uint2(0u, 0u);
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  const bool issuer = warp == 0;
  float acc[NY / 2] = {};
  for (int half = 0; half < 2; ++half) {
    const int t0 = half * 64;
    if (half == 1 && n <= 64) break;
    if (half == 1 && __syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    auto tile = [&](auto t, unsigned char* to, auto at, auto scale) {
      using T = decltype(t);
      constexpr int U = 4;
#pragma unroll
      for (int i0 = 0; i0 < T::PIECES; i0 += U) {
        float4 v[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int row = t0 + T::row(i0 + i);
          v[i] = row < n ? *reinterpret_cast<const float4*>(at((size_t)(first + row)) + T::col()) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const float2 f = scale(t0 + T::row(i0 + i));
          v[i].x *= f.x; v[i].y *= f.x; v[i].z *= f.x; v[i].w *= f.x;
          largest = tc_largest(largest, v[i]);
          v[i].x *= f.y; v[i].y *= f.y; v[i].z *= f.y; v[i].w *= f.y;
          tc_put<64, T::ACROSS * 4>(to, T::row(i0 + i), T::col(), v[i]);
        }
      }
    };
    auto keys = [&](size_t row) { return a.k + row * a.k_stride + (size_t)g * DK; };
    auto values = [&](size_t row) { return a.v + row * a.v_stride + (size_t)h * DV; };
    // a key's step, as the scan has it (which may go beyond float32), then the decays behind it
    auto key_scale = [&](int row) { return make_float2(MODE == CHUNK_STEP ? decay.step[row] : 1.0f, row < n ? decay.between(row + 1, n) : 1.0f); };
    auto one = [](int) { return make_float2(1.0f, 1.0f); };
    if (DK == 128) {
      tile(TcTile<64, 128, 256>(), smem, keys, key_scale);
      tile(TcTile<64, NY, 256>(), smem + L::X, values, one);
    } else {
      tile(TcTile<64, 128, 256>(), smem, values, one);
      tile(TcTile<64, NY, 256>(), smem + L::X, keys, key_scale);
    }
    fence_proxy_async_smem();
    bad = __syncthreads_or(bad || largest >= kTcCut);
    if (bad) break;
    const uint64_t xd = tc_mn_major(x0, 64 * 128), yd = tc_mn_major(y0, 64 * 128);
    auto x = [&](int p, int ks) { return xd + ((p * (2 * 64 * 128) + ks * 2048) >> 4); };
    auto y = [&](int p, int ks) { return yd + ((p * (NY / 64 * 64 * 128) + ks * 2048) >> 4); };
    ok = tc_product<NY, 4, L::SLOTS>(acc, tmem, lanes + (warp >> 2) * (NY / 2), bar, phase, issuer, x, y,
                                     [&](uint32_t d, uint64_t xa, uint64_t yb, uint32_t on, uint32_t elected) { umma_ss(d, xa, yb, tc_idesc(NY, 1, 1), on, elected); },
                                     half == 1, [] {});
  }
  float* local = a.local + item * DV * DK;
  ok = !__syncthreads_or(!ok);
  if (bad) {                                               // token by token, a thread per value channel
    if (ok && (int)threadIdx.x < DV) {
      float S[DK];                                         // in local memory: this path is for correctness
#pragma unroll 1
      for (int c = 0; c < DK; ++c) S[c] = 0.0f;
#pragma unroll 1
      for (int t = 0; t < n; ++t) {
        const size_t row = (size_t)(first + t);
        const float v = a.v[row * a.v_stride + (size_t)h * DV + threadIdx.x], st = MODE == CHUNK_STEP ? decay.step[t] : 1.0f;
        const float w = MODE == CHUNK_STEP ? expf(-expf(a.log_rate[h]) * st) : a.rate[h];
#pragma unroll 1
        for (int c = 0; c < DK; ++c) S[c] = fmaf(w, S[c], a.k[row * a.k_stride + (size_t)g * DK + c] * st * v);
      }
#pragma unroll 1
      for (int c = 0; c < DK; ++c) local[(size_t)threadIdx.x * DK + c] = S[c];
    }
  } else if (ok) {
    tc_add_small(acc, tmem, lanes + (warp >> 2) * (NY / 2));
    const int row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * (NY / 2);
    if (DK == 128) {
      {
#pragma unroll
        for (int i = 0; i < NY / 2; ++i) local[(size_t)(c0 + i) * DK + row] = acc[i];
      }
    } else {                                               // rows of 64 through shared memory: whole ones to a store instruction
      constexpr int PITCH = NY + 4;
      float* rows = reinterpret_cast<float*>(smem);
      {
#pragma unroll
        for (int i = 0; i < NY / 2; i += 4)
          *reinterpret_cast<float4*>(rows + row * PITCH + c0 + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
      }
      __syncthreads();
#pragma unroll 4
      for (int e = threadIdx.x * 4; e < 128 * NY; e += 256 * 4)
        *reinterpret_cast<float4*>(local + e) = *reinterpret_cast<const float4*>(rows + e / NY * PITCH + e % NY);
    }
  }
  if (!ok && lane == 0) atomicExch(error_flag, 81);
  tc_before();
  __syncthreads();
  if (warp == 0) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)L::COLUMNS) : "memory");
  }
}

// -------------------------------------------------------------------------------------------- outputs
// A block takes `each` heads that share queries and keys, whose scores it makes once.  Two places for operands: queries, then (values of
// 128) values; keys, then the state in front and (values of 64) values, or scores times decays.  With values of 64 the parts of scores
// times decays go to tensor memory, columns 0 .. 191, and accumulators lie behind them.
template <int DK, int DV>
struct TcOut {
  static constexpr int THREADS = 512;
  static constexpr bool IN_TMEM = DV == 64;
  static constexpr uint32_t Q = TcTile<kTc, DK, THREADS>::BYTES, V = TcTile<kTc, DV, THREADS>::BYTES, S = TcTile<DV, DK, THREADS>::BYTES,
                            P = TcTile<kTc, kTc, THREADS>::BYTES, BEHIND = IN_TMEM ? S + V : P;
  static constexpr uint32_t FIRST = IN_TMEM || Q > V ? Q : V, SECOND = Q > BEHIND ? Q : BEHIND;
  static constexpr uint32_t AT = IN_TMEM ? 192 : 0;
  static constexpr int SLOTS = (512 - AT) / DV;
  static constexpr size_t SMEM = 1024 + FIRST + SECOND;
};

template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(512, 1) chunk_outputs_kernel(const ChunkArgs a, int each, int* error_flag) {
  using L = TcOut<DK, DV>;
  using TQ = TcTile<kTc, DK, 512>;
  using TV = TcTile<kTc, DV, 512>;
  using TS = TcTile<DV, DK, 512>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ TcDecay<MODE> decay;
  __shared__ uint64_t bar_s[2];
  __shared__ uint32_t tmem_holder;
  const int g = blockIdx.y * each / (a.heads / a.groups);
  int first, n;
  if (!chunk_of(a.cu_seqlens, a.requests, a.min_span, blockIdx.x, first, n, kTc)) return;
  unsigned char* one = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  unsigned char* two = one + L::FIRST;
  unsigned char* values = L::IN_TMEM ? two + L::S : one;
  const uint32_t a0 = smem_addr(one), b0 = smem_addr(two), v0 = smem_addr(values), bar = smem_addr(bar_s);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const bool issuer = warp == 0;
  uint32_t largest = 0;
  {
    constexpr int U = TQ::PIECES;
#pragma unroll
    for (int i0 = 0; i0 < TQ::PIECES; i0 += U) {
      float4 q[U], k[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int t = TQ::row(i0 + i);
        const size_t row = (size_t)(first + t);
        q[i] = t < n ? *reinterpret_cast<const float4*>(a.q + row * a.q_stride + (size_t)g * DK + TQ::col()) : none;
        k[i] = t < n ? *reinterpret_cast<const float4*>(a.k + row * a.k_stride + (size_t)g * DK + TQ::col()) : none;
      }
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int t = TQ::row(i0 + i);
        q[i].x *= a.q_scale; q[i].y *= a.q_scale; q[i].z *= a.q_scale; q[i].w *= a.q_scale;
        largest = tc_largest(tc_largest(largest, q[i]), k[i]);
        if (MODE == CHUNK_STEP) {
          const unsigned row_lanes = TQ::ACROSS == 32 ? 0xffffffffu : 0xffffu << (threadIdx.x & 16);
          decay.key[t] = __uint_as_float(__reduce_max_sync(row_lanes, tc_largest(0u, k[i])));
        }
        tc_put<kTc, DK>(one, t, TQ::col(), q[i]);
        tc_put<kTc, DK>(two, t, TQ::col(), k[i]);
      }
    }
  }
  fence_proxy_async_smem();
  tc_before();
  const bool bad_rows = __syncthreads_or(largest >= kTcCut);
  tc_after();
  const uint32_t tmem = tmem_holder;
  bool ok = true;
  const int row = (warp & 3) * 32 + lane, quarter = warp >> 2;               // this thread's token and quarter of the columns
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  uint2 phase = make_uint2(0u, 0u);
  constexpr uint32_t kHalf = kTc * 128;
  // operands: a descriptor and, added to its address, constants (the whole of shared memory fits the field)
  const uint64_t d_one = tc_k_major(a0), d_two = tc_k_major(b0), d_values = tc_mn_major(v0, kHalf);
  auto q_k = [&](int p, int ks) { return d_one + ((p * TQ::PART + (ks >> 2) * kHalf + (ks & 3) * 32) >> 4); };
  float scores[32] = {};
  bool bad_decay = false;
  auto state_of = [&](int h) { return a.local + ((size_t)blockIdx.x * a.heads + h) * DV * DK; };
  const int h0 = blockIdx.y * each;
  if (bad_rows) bad_decay = decay.make(a, h0, first, n);
  if (!bad_rows) {
    auto k_k = [&](int p, int ks) { return d_two + ((p * TQ::PART + (ks >> 2) * kHalf + (ks & 3) * 32) >> 4); };
    ok = tc_product<kTc, DK / 16, 4>(scores, tmem, lanes + quarter * 32, bar, phase, issuer, q_k, k_k,
                                     [&](uint32_t d, uint64_t x, uint64_t y, uint32_t on, uint32_t elected) { umma_ss(d, x, y, tc_idesc(kTc, 0, 0), on, elected); },
                                     false, [&] {
      bad_decay = decay.make(a, h0, first, n);
    });
    tc_add_small(scores, tmem, lanes + quarter * 32);
  }
  for (int h = h0; h < h0 + each; ++h) {
    ok = !__syncthreads_or(!ok);                           // the head before is done with everything
    if (!ok) break;
    const float* state = state_of(h);
    // four pieces a thread at a time, which are all with values of 64
    auto move_v = [&]() {
#pragma unroll
      for (int i0 = 0; i0 < TV::PIECES; i0 += 4) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = TV::row(i0 + i);
          v[i] = t < n ? *reinterpret_cast<const float4*>(a.v + (size_t)(first + t) * a.v_stride + (size_t)h * DV + TV::col()) : none;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          largest = tc_largest(largest, v[i]);
          tc_put<kTc, DV>(values, TV::row(i0 + i), TV::col(), v[i]);
        }
      }
    };
    largest = 0;
    if (!bad_rows) {
#pragma unroll
      for (int i0 = 0; i0 < TS::PIECES; i0 += 4) {
        float4 s[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = *reinterpret_cast<const float4*>(state + (size_t)TS::row(i0 + i) * DK + TS::col());
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          largest = tc_largest(largest, s[i]);
          tc_put<DV, DK>(two, TS::row(i0 + i), TS::col(), s[i]);
        }
      }
      if (L::IN_TMEM) move_v();
    }
    if (h > h0) bad_decay = decay.make(a, h, first, n);
    if (MODE == CHUNK_STEP && threadIdx.x < kTc) largest = max(largest, magnitude(decay.key[threadIdx.x] * decay.step[threadIdx.x]));
    bool bad = bad_decay || bad_rows;
    float out[DV / 4] = {};
    fence_proxy_async_smem();
    bad = __syncthreads_or(bad || largest >= kTcCut);
    if (!bad) {
      // scores times decays (and steps): columns quarter * 32 + 16 j .. + 15 of this token's row
      auto weighed = [&](int j, float (&w)[16]) {
        const int k0 = quarter * 32 + j * 16, behind = k0 + 16;
        if (MODE == CHUNK_STEP) {
          // pairs further apart by way of the end of the 16 columns; decays within the row's own 16 one by one
          const float to = behind <= row ? decay.between(behind, row + 1) : 0.0f;
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = to * decay.rest[k0 + i];
          const bool own = (row >> 4) == (k0 >> 4);
          if (__any_sync(0xffffffffu, own)) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int k = k0 + i;
              const float d = decay.between(min(k, row) + 1, row + 1) * decay.step[k];
              w[i] = own ? d : w[i];
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = decay.between(min(k0 + i, row) + 1, row + 1);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          w[i] = k0 + i <= row ? scores[16 * j + i] * w[i] : 0.0f;
          largest = max(largest, magnitude(w[i]));
        }
      };
      auto s_k = [&](int p, int ks) { return d_two + ((p * TS::PART + (ks >> 2) * (DV * 128) + (ks & 3) * 32) >> 4); };
      ok = tc_product<DV, DK / 16, L::SLOTS>(out, tmem + L::AT, lanes + quarter * (DV / 4), bar, phase, issuer, q_k, s_k,
                                             [&](uint32_t d, uint64_t x, uint64_t y, uint32_t on, uint32_t elected) { umma_ss(d, x, y, tc_idesc(DV, 0, 0), on, elected); },
                                             false, [&]() {
        if constexpr (L::IN_TMEM) {
          uint32_t pairs[3][16];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            float w[16];
            weighed(j, w);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const Cut cut(w[2 * i], w[2 * i + 1]);
#pragma unroll
              for (int p = 0; p < 3; ++p) pairs[p][8 * j + i] = cut.part[p];
            }
          }
#pragma unroll
          for (int p = 0; p < 3; ++p) tc_st16(tmem + lanes + p * 64 + quarter * 16, pairs[p]);
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            float w[16];
            weighed(j, w);
#pragma unroll
            for (int i = 0; i < 16; ++i) scores[16 * j + i] = w[i];
          }
          // 512 lines of values, one a thread, come nearer
          const int t = threadIdx.x >> 2;
          if (t < n)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.v + (size_t)(first + t) * a.v_stride + (size_t)h * DV + (threadIdx.x & 3) * 32));
        }
      });
      tc_add_small(out, tmem + L::AT, lanes + quarter * (DV / 4));
      const float f = decay.between(0, min(row, n - 1) + 1);
#pragma unroll
      for (int i = 0; i < DV / 4; ++i) out[i] *= f;
      if constexpr (!L::IN_TMEM) {
        // (the products of queries have ended in every thread's eyes: `one` and `two` are free)
        move_v();
#pragma unroll
        for (int c = 0; c < 4; ++c) {                      // eight columns, 16 bytes of a part
          const Cut c0(scores[8 * c], scores[8 * c + 1]), c1(scores[8 * c + 2], scores[8 * c + 3]), c2(scores[8 * c + 4], scores[8 * c + 5]),
              c3(scores[8 * c + 6], scores[8 * c + 7]);
          const int piece = quarter * 4 + c;
          unsigned char* at = two + (piece >> 3) * kHalf + row * 128 + (((piece & 7) ^ (row & 7)) << 4);
#pragma unroll
          for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(at + p * 2 * kHalf) = make_uint4(c0.part[p], c1.part[p], c2.part[p], c3.part[p]);
        }
        fence_proxy_async_smem();
      }
      tc_before();
      bad = __syncthreads_or(largest >= kTcCut);
      if (!bad) {                                          // the sums of values
        auto v_mn = [&](int p, int ks) { return d_values + ((p * TV::PART + ks * 2048) >> 4); };
        bool done;
        float sums[DV / 4] = {};
        if constexpr (L::IN_TMEM) {
          auto p_t = [&](int p, int ks) { return tmem + p * 64 + ks * 8; };
          done = tc_product<DV, kTc / 16, L::SLOTS>(sums, tmem + L::AT, lanes + quarter * (DV / 4), bar, phase, issuer, p_t, v_mn,
                                                    [&](uint32_t d, uint32_t x, uint64_t y, uint32_t on, uint32_t elected) {
                                                      umma_ts(d, x, y, tc_idesc(DV, 0, 1), on, elected);
                                                    }, false, [] {});
        } else {
          auto p_k = [&](int p, int ks) { return d_two + ((p * 2 * kHalf + (ks >> 2) * kHalf + (ks & 3) * 32) >> 4); };
          done = tc_product<DV, kTc / 16, L::SLOTS>(sums, tmem + L::AT, lanes + quarter * (DV / 4), bar, phase, issuer, p_k, v_mn,
                                                    [&](uint32_t d, uint64_t x, uint64_t y, uint32_t on, uint32_t elected) {
                                                      umma_ss(d, x, y, tc_idesc(DV, 0, 1), on, elected);
                                                    }, false, [] {});
        }
        ok = done && ok;
        tc_add_small(sums, tmem + L::AT, lanes + quarter * (DV / 4));
#pragma unroll
        for (int i = 0; i < DV / 4; ++i) out[i] += sums[i];
      }
    }
    const float skip = a.skip ? a.skip[h] : 0.0f;
    if (bad) {                                             // token by token from the state in front, a thread per value channel
      if ((int)threadIdx.x < DV) {
        float S[DK];                                       // in local memory: this path is for correctness
#pragma unroll 1
        for (int c = 0; c < DK; ++c) S[c] = state[(size_t)threadIdx.x * DK + c];
#pragma unroll 1
        for (int t = 0; t < n; ++t) {
          const size_t at = (size_t)(first + t);
          const float value = a.v[at * a.v_stride + (size_t)h * DV + threadIdx.x], st = MODE == CHUNK_STEP ? decay.step[t] : 1.0f;
          const float w = MODE == CHUNK_STEP ? expf(-expf(a.log_rate[h]) * st) : a.rate[h];
          float acc = 0.0f;
#pragma unroll 1
          for (int c = 0; c < DK; ++c) {
            S[c] = fmaf(w, S[c], a.k[at * a.k_stride + (size_t)g * DK + c] * st * value);
            acc = fmaf(a.q[at * a.q_stride + (size_t)g * DK + c] * a.q_scale, S[c], acc);
          }
          a.out[at * a.heads * DV + (size_t)h * DV + threadIdx.x] = a.skip ? fmaf(skip, value, acc) : acc;
        }
      }
    } else {
      // through shared memory (`two` is free): whole rows to a store instruction instead of 16 bytes of 32 rows
      constexpr int PITCH = DV + 4;
      float* rows = reinterpret_cast<float*>(two);
      {
#pragma unroll
        for (int i = 0; i < DV / 4; i += 4)
          *reinterpret_cast<float4*>(rows + row * PITCH + quarter * (DV / 4) + i) = make_float4(out[i], out[i + 1], out[i + 2], out[i + 3]);
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < TV::PIECES; ++i) {
        const int t = TV::row(i), c = TV::col();
        if (t >= n || !ok) continue;
        const size_t at = (size_t)(first + t);
        float4 o = *reinterpret_cast<const float4*>(rows + t * PITCH + c);
        if (a.skip) {
          const float4 x = *reinterpret_cast<const float4*>(a.v + at * a.v_stride + (size_t)h * DV + c);
          o.x = fmaf(skip, x.x, o.x); o.y = fmaf(skip, x.y, o.y); o.z = fmaf(skip, x.z, o.z); o.w = fmaf(skip, x.w, o.w);
        }
        *reinterpret_cast<float4*>(a.out + at * a.heads * DV + (size_t)h * DV + c) = o;
      }
    }
  }
  if (!ok && lane == 0) atomicExch(error_flag, 82);
  tc_before();
  __syncthreads();
  if (warp == 0) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

int launch_chunk_carry(const ChunkArgs& a, int dk, cudaStream_t stream);      // chunk_scan.cu

template <int DK, int DV, int MODE>
static int launch_tc(const ChunkArgs& a, int chunks, int* error_flag, cudaStream_t stream) {
  auto add = chunk_add_kernel<DK, DV, MODE>;
  auto outputs = chunk_outputs_kernel<DK, DV, MODE>;
  cudaError_t e = cudaFuncSetAttribute(add, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TcAdd<DK, DV>::SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(outputs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TcOut<DK, DV>::SMEM);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid(chunks, a.heads);
  add<<<grid, 256, TcAdd<DK, DV>::SMEM, stream>>>(a, error_flag);
  IFX_CHECK_LAUNCH();
  const int rc = launch_chunk_carry(a, DK, stream);
  if (rc) return rc;
  // Heads that share queries and keys go together where that takes less: a block's scores cost about three fifths of a head.  (24 heads,
  // 2,048 tokens: 408 blocks of a head in three rounds, or 136 of three in one; 56 heads, 300 tokens: 168 and two rounds, or 84.)
  const int share = TcOut<DK, DV>::IN_TMEM ? a.heads / a.groups : 1;
  int each = 1;
  long long least = 0;
  for (int e = 1; e <= 4; ++e) {
    if (share % e) continue;
    const long long cost = ((long long)chunks * (a.heads / e) + 147) / 148 * (3 + 5 * e);
    if (e == 1 || cost < least) each = e, least = cost;
  }
  outputs<<<dim3(chunks, a.heads / each), 512, TcOut<DK, DV>::SMEM, stream>>>(a, each, error_flag);
  IFX_CHECK_LAUNCH();
  return 0;
}

// Heads of 64 x 64 have no side of 128 for a product's rows: they go by stretches of 64.
bool chunks_of_128_take(int mode, int dk, int dv) {
  return (mode == CHUNK_STEP || mode == CHUNK_CONSTANT) && ((dk == 128 && (dv == 64 || dv == 128)) || (dk == 64 && dv == 128));
}

int launch_chunks_of_128(const ChunkArgs& a, int dk, int mode, int chunks, int* error_flag, cudaStream_t stream) {
  if (mode == CHUNK_STEP) {
    if (dk == 128 && a.dv == 128) return launch_tc<128, 128, CHUNK_STEP>(a, chunks, error_flag, stream);
    if (dk == 128 && a.dv == 64) return launch_tc<128, 64, CHUNK_STEP>(a, chunks, error_flag, stream);
    if (dk == 64 && a.dv == 128) return launch_tc<64, 128, CHUNK_STEP>(a, chunks, error_flag, stream);
  } else if (mode == CHUNK_CONSTANT) {
    if (dk == 128 && a.dv == 128) return launch_tc<128, 128, CHUNK_CONSTANT>(a, chunks, error_flag, stream);
    if (dk == 128 && a.dv == 64) return launch_tc<128, 64, CHUNK_CONSTANT>(a, chunks, error_flag, stream);
    if (dk == 64 && a.dv == 128) return launch_tc<64, 128, CHUNK_CONSTANT>(a, chunks, error_flag, stream);
  }
  return IFX_E_BADARG;
}

}  // namespace ifx
