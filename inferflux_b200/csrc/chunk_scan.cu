// The scans of decay_scan.cu and wkv.cu over long spans, a stretch of 64 tokens at a time instead of token after token.  (One decay
// per head with keys or values of 128: chunk_tcgen05.cu, 128 tokens at a time, with this file's carry.)
// With S_0 the state in front of a stretch, and products of decays w over the tokens between,
//
//   o_t  = (q_t * prod w_1..t)^T S_0  +  sum over s <= t of (q_t . (k_s * prod w_s+1..t)) v_s
//   S_64 = diag(prod w_1..64) S_0     +  sum over s of (k_s * prod w_s+1..64) v_s^T
//
// (wkv: the decays up to t - 1 and s < t, the present token with the bonus u in place of a decay.)  Three kernels:
//
//   chunk_local   per stretch, head and 64 value channels, without S_0: the second sum of o_t, the second term of S_64, the
//                 products of decays that the next two need
//   chunk_carry   the states in front of every stretch, element by element along a request
//   chunk_reach   adds the first term of o_t
//
// so that every SM works on a prompt whose tokens a scan takes one after the other.  Nothing is divided by a decay and no
// logarithm is taken: products of decays are multiplied up, so a decay may be zero and the error is that of the scan.
// With a decay per key channel, pairs (t, s) within 16 tokens are multiplied up one by one; for pairs further apart the
// product is cut at the beginnings of the 16s, q_t taking what lies in its own 16, k_s the rest of its own, and whole 16s
// between as factors.  Matrix products run on the tensor cores with both operands split into three (chunk_scan.cuh).
//
// A stretch that holds a number that is not finite, or in which the product of a query and a key is none, is walked token by
// token by its block, so that such a number reaches what it would reach in a scan and nothing in front of it, and so that a product
// that a scan would not have formed spoils nothing.
//
// The order of the sums depends on where a span is cut into steps, so the float32 run keeps the scans.
//
// Bound: no unit alone.  chunk_local splits every operand into three and makes eight products of them: issue slots 44 % busy, ALU 35 %,
// tensor pipe 31 %, with 14 warps an SM that wait for barriers, for the latency of that chain and for states, which go through L2
// twice (26 MB at 2,048 tokens of 12 heads of 128 x 128).  A warp's tile is 32 x 16, so that an operand is split and read
// by few warps.  Measured, us, scan -> this, one span of 2,048 tokens: constant decay, 12 heads of 128 x 128 590 -> 120; wkv, 24
// heads of 64 (with its norm) 521 -> 127; a decay per token, 24 heads of 128 x 64 693 -> 117; per key channel, 12 heads of
// 64 x 128 491 -> 93.  At 130 tokens 42 -> 32, 41 -> 30, 50 -> 32, 36 -> 25; at 64 the scan is the faster.
// Errors of outputs and of the state against 64 bits (2-norm, scan and this, parameters where trained models have them, 2,048
// tokens): constant decay 3.5e-7 and 1.1e-7, 3.8e-7 and 0.8e-7; a decay per token 1.65e-7 and 1.53e-7, 1.30e-7 and 1.22e-7; per key
// channel 3.20e-6 and 3.16e-6, 3.98e-6 and 3.96e-6; wkv's state 9.14e-7 and 9.17e-7.  (With operands of 22 bits and sums left in the
// tensor cores' accumulators it was 15, 9.8, 2.9 and 8.9e-7, a fifth faster.)
#include "chunk_scan.cuh"

namespace ifx {

template <int DK, int MODE>
struct ChunkLayout {
  static constexpr bool CHANNEL = MODE == CHUNK_CHANNEL || MODE == CHUNK_WKV;
  static constexpr int PK = DK + 8;
  static constexpr int Q = 0, K = Q + kChunk * PK, V = K + kChunk * PK, A = V + kChunk * kPitchV, W = A + kChunk * kPitchA,
                       SMALL = W + (CHANNEL ? kChunk * PK : 0);          // CHANNEL: decays of the 16s [4][DK]; else w, step, tail [64] each
  static constexpr size_t BYTES = (size_t)(SMALL + (CHANNEL ? 4 * DK : 3 * kChunk)) * sizeof(float);
};

template <int DK, int MODE>
__global__ void __launch_bounds__(256) chunk_local_kernel(const ChunkArgs a) {
  using L = ChunkLayout<DK, MODE>;
  constexpr int PK = L::PK;
  extern __shared__ __align__(16) float smem[];
  float *q_s = smem + L::Q, *k_s = smem + L::K, *v_s = smem + L::V, *a_s = smem + L::A, *w_s = smem + L::W, *small = smem + L::SMALL;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, z = blockIdx.z, g = h / (a.heads / a.groups), dv = a.dv;
  int first, n;
  if (!chunk_of(a.cu_seqlens, a.requests, a.min_span, blockIdx.x, first, n)) return;
  const size_t item = (size_t)blockIdx.x * a.heads + h;

  if (!L::CHANNEL) {                                       // decays and steps of the tokens; rows behind the last leave the state alone
    if (tid < kChunk) {
      float w = 1.0f, step = 1.0f;
      if (tid < n) {
        if (MODE == CHUNK_STEP) {
          step = chunk_softplus(a.raw[(size_t)(first + tid) * a.raw_stride + h] + a.step_bias[h]);
          w = expf(-expf(a.log_rate[h]) * step);
        } else {
          w = a.rate[h];
        }
      }
      small[tid] = w;
      small[kChunk + tid] = step;
    }
    __syncthreads();
  }
  bool bad = !L::CHANNEL && tid < kChunk && !splits(small[tid]);
  for (int e = tid; e < kChunk * DK / 4; e += 256) {
    const int t = e / (DK / 4), c = e % (DK / 4) * 4;
    const size_t row = (size_t)(first + t);
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f), k = q, w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    if (t < n) {
      q = *reinterpret_cast<const float4*>(a.q + row * a.q_stride + (size_t)g * DK + c);
      k = *reinterpret_cast<const float4*>(a.k + row * a.k_stride + (size_t)g * DK + c);
      q.x *= a.q_scale; q.y *= a.q_scale; q.z *= a.q_scale; q.w *= a.q_scale;
      if (MODE == CHUNK_STEP) {
        const float step = small[kChunk + t];
        k.x *= step; k.y *= step; k.z *= step; k.w *= step;
      }
      if (L::CHANNEL) {
        const float4 r = *reinterpret_cast<const float4*>(a.raw + row * a.raw_stride + (size_t)h * DK + c);
        if (MODE == CHUNK_CHANNEL) {
          w.x = expf(chunk_log_sigmoid(r.x) * a.inv_tau); w.y = expf(chunk_log_sigmoid(r.y) * a.inv_tau);
          w.z = expf(chunk_log_sigmoid(r.z) * a.inv_tau); w.w = expf(chunk_log_sigmoid(r.w) * a.inv_tau);
        } else {
          const float4 w0 = *reinterpret_cast<const float4*>(a.w0 + (size_t)h * DK + c);
          w.x = expf(-expf(r.x + w0.x)); w.y = expf(-expf(r.y + w0.y));
          w.z = expf(-expf(r.z + w0.z)); w.w = expf(-expf(r.w + w0.w));
        }
        bad = bad || !splits(w);
      }
    }
    bad = bad || !splits(q) || !splits(k);
    *reinterpret_cast<float4*>(q_s + t * PK + c) = q;
    *reinterpret_cast<float4*>(k_s + t * PK + c) = k;
    if (L::CHANNEL) *reinterpret_cast<float4*>(w_s + t * PK + c) = w;
  }
  for (int e = tid; e < kChunk * 16; e += 256) {
    const int t = e >> 4, c = (e & 15) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < n) v = *reinterpret_cast<const float4*>(a.v + (size_t)(first + t) * a.v_stride + (size_t)h * dv + z * 64 + c);
    bad = bad || !splits(v);
    *reinterpret_cast<float4*>(v_s + t * kPitchV + c) = v;
  }
  bad = __syncthreads_or(bad);

  uint32_t largest = 0;                                    // of what is made here to be split
  // ---------------------------------------------------------- decays multiplied up; pairs of tokens within 16
  if (L::CHANNEL && !bad) {
    const int i = tid >> 6, s = (tid >> 2) & 15, part = tid & 3, tok = i * kSub + s;       // four lanes share a key
    float kp[DK / 4];
#pragma unroll
    for (int m = 0; m < DK / 16; ++m) {
      const float4 k4 = *reinterpret_cast<const float4*>(k_s + tok * PK + 16 * m + 4 * part);
      kp[4 * m] = k4.x; kp[4 * m + 1] = k4.y; kp[4 * m + 2] = k4.z; kp[4 * m + 3] = k4.w;
    }
    for (int t = 0; t < kSub; ++t) {
      const int row = i * kSub + t;
      float acc = 0.0f;
#pragma unroll
      for (int m = 0; m < DK / 16; ++m) {
        const int c = 16 * m + 4 * part;
        float4 q4 = *reinterpret_cast<const float4*>(q_s + row * PK + c);
        const float4 w4 = *reinterpret_cast<const float4*>(w_s + row * PK + c);
        float f[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = t > s ? f[e] : 1.0f;
        if (MODE == CHUNK_WKV && t == s) {
          const float4 u4 = *reinterpret_cast<const float4*>(a.u + (size_t)h * DK + c);
          q4.x *= u4.x; q4.y *= u4.y; q4.z *= u4.z; q4.w *= u4.w;
        }
        if (MODE == CHUNK_CHANNEL) {
#pragma unroll
          for (int e = 0; e < 4; ++e) kp[4 * m + e] *= f[e];
        }
        acc = fmaf(q4.x, kp[4 * m], acc);
        acc = fmaf(q4.y, kp[4 * m + 1], acc);
        acc = fmaf(q4.z, kp[4 * m + 2], acc);
        acc = fmaf(q4.w, kp[4 * m + 3], acc);
        if (MODE == CHUNK_WKV) {
#pragma unroll
          for (int e = 0; e < 4; ++e) kp[4 * m + e] *= f[e];
        }
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc = t >= s ? acc : 0.0f;
      largest = max(largest, magnitude(acc));
      if (part == 0) a_s[row * kPitchA + tok] = acc;
    }
    __syncthreads();
  }
  if (L::CHANNEL) {                                        // (a stretch with bad numbers needs the totals and reaches too)
    for (int e = tid; e < 4 * DK; e += 256) {
      const int i = e / DK, c = e % DK;
      float p = 1.0f;
#pragma unroll
      for (int t = 0; t < kSub; ++t) {
        float* qp = q_s + (i * kSub + t) * PK + c;
        const float w = w_s[(i * kSub + t) * PK + c];
        if (MODE == CHUNK_WKV) { if (!bad) *qp *= p; p *= w; }
        else { p *= w; if (!bad) *qp *= p; }
      }
      small[i * DK + c] = p;
      float rest = 1.0f;
#pragma unroll
      for (int t = kSub - 1; t >= 0; --t) {
        if (!bad) k_s[(i * kSub + t) * PK + c] *= rest;
        rest *= w_s[(i * kSub + t) * PK + c];
      }
    }
    __syncthreads();
    if (z == 0) {
      if (!bad) {
        for (int e = tid; e < n * (DK / 4); e += 256) {
          const int t = e / (DK / 4), c = e % (DK / 4) * 4;
          float4 q = *reinterpret_cast<const float4*>(q_s + t * PK + c);
          for (int j = 0; j < t / kSub; ++j) {
            const float4 f = *reinterpret_cast<const float4*>(small + j * DK + c);
            q.x *= f.x; q.y *= f.y; q.z *= f.z; q.w *= f.w;
          }
          *reinterpret_cast<float4*>(a.reach + (size_t)(first + t) * a.heads * DK + (size_t)h * DK + c) = q;
        }
      } else {
        for (int c = tid; c < DK; c += 256) {
          float p = 1.0f;
          for (int t = 0; t < n; ++t) {
            if (MODE != CHUNK_WKV) p *= w_s[t * PK + c];
            a.reach[(size_t)(first + t) * a.heads * DK + (size_t)h * DK + c] = q_s[t * PK + c] * p;
            if (MODE == CHUNK_WKV) p *= w_s[t * PK + c];
          }
        }
      }
      for (int c = tid; c < DK; c += 256) a.total[item * DK + c] = small[c] * small[DK + c] * small[2 * DK + c] * small[3 * DK + c];
    }
  } else {
    if (tid < kChunk) {                                    // column s of the decays from s + 1 to t
      Product p;
      for (int t = tid; t < kChunk; ++t) {
        if (t > tid) p.times(small[t]);
        a_s[t * kPitchA + tid] = p.value();
      }
      small[2 * kChunk + tid] = p.value();                 // to the end
      largest = magnitude(p.value());
      if (tid == 0 && z == 0) {
        p.times(small[0]);
        a.total[2 * item] = p.value();
        a.total[2 * item + 1] = (p.hi - p.value()) + p.lo;
      }
    }
    __syncthreads();
    if (z == 0) {
      if (tid < n) a.reach[(size_t)(first + tid) * a.heads + h] = a_s[tid * kPitchA] * small[0];
      __syncthreads();                                     // read, before the products below go over it
    }
  }
  float* out = a.out + (size_t)first * a.heads * dv + (size_t)h * dv + z * 64;
  const size_t out_row = (size_t)a.heads * dv;
  float* local = a.local + (item * dv + z * 64) * DK;
  const float skip = a.skip ? a.skip[h] : 0.0f;

  // ---------------------------------------------------------- pairs of tokens: 16 x 8 tiles of q . k
  if (!bad && L::CHANNEL) {
    for (int task = warp; task < 12; task += 8) {          // (i, j < i, half): rows of the i-th 16, columns of the j-th
      const int pair = task >> 1, i = pair == 0 ? 1 : pair < 3 ? 2 : 3, j = pair == 0 ? 0 : pair < 3 ? pair - 1 : pair - 3;
      const int r0 = i * kSub, c0 = j * kSub + (task & 1) * 8;
      float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
      for (int kk = 0; kk < DK; kk += 16) {
        FragA fa;
        FragB fb;
        load_a_rows(fa, q_s + r0 * PK + kk, PK, lane);
        float2 b[2] = {read_b_rows(k_s + c0 * PK + kk, PK, lane), read_b_rows(k_s + c0 * PK + kk + 8, PK, lane)};
        for (int m = j + 1; m < i; ++m) {
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const float2 f = *reinterpret_cast<const float2*>(small + m * DK + kk + 8 * x + 2 * (lane & 3));
            b[x].x *= f.x;
            b[x].y *= f.y;
          }
        }
        fb.v[0].set(b[0].x, b[1].x);
        fb.v[1].set(b[0].y, b[1].y);
        mma_split(c, fa, fb);
      }
      float* to = a_s + (r0 + (lane >> 2)) * kPitchA + c0 + 2 * (lane & 3);
      to[0] = c[0];
      to[1] = c[1];
      to[8 * kPitchA] = c[2];
      to[8 * kPitchA + 1] = c[3];
#pragma unroll
      for (int i = 0; i < 4; ++i) largest = max(largest, magnitude(c[i]));
    }
  } else if (!bad) {
    for (int task = warp; task < 20; task += 8) {          // the tiles at and below the diagonal
      const int i = task < 2 ? 0 : task < 6 ? 1 : task < 12 ? 2 : 3;
      const int r0 = i * kSub, c0 = (task - i * (i + 1)) * 8;
      float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
      for (int kk = 0; kk < DK; kk += 16) {
        FragA fa;
        FragB fb;
        load_a_rows(fa, q_s + r0 * PK + kk, PK, lane);
        load_b_rows(fb, k_s + c0 * PK + kk, PK, lane);
        mma_split(c, fa, fb);
      }
      const int t = r0 + (lane >> 2), s = c0 + 2 * (lane & 3);
      float* to = a_s + t * kPitchA + s;
      c[0] = s <= t ? to[0] * c[0] : 0.0f;
      c[1] = s + 1 <= t ? to[1] * c[1] : 0.0f;
      c[2] = s <= t + 8 ? to[8 * kPitchA] * c[2] : 0.0f;
      c[3] = s + 1 <= t + 8 ? to[8 * kPitchA + 1] * c[3] : 0.0f;
      to[0] = c[0];
      to[1] = c[1];
      to[8 * kPitchA] = c[2];
      to[8 * kPitchA + 1] = c[3];
#pragma unroll
      for (int i = 0; i < 4; ++i) largest = max(largest, magnitude(c[i]));
    }
  }
  bad = __syncthreads_or(bad || largest >= kSplitLimit);
  if (bad) {                                               // token by token, a thread per value channel (CHANNEL: q_s, k_s may be scaled)
    if (tid < 64) {
      float S[DK];                                         // in local memory: this path is for correctness
#pragma unroll 1
      for (int c = 0; c < DK; ++c) S[c] = 0.0f;
      for (int t = 0; t < n; ++t) {
        const float v = v_s[t * kPitchV + tid];
        float acc = 0.0f, bonus = 0.0f;
#pragma unroll 1
        for (int c = 0; c < DK; ++c) {
          const float q = L::CHANNEL ? a.q[(size_t)(first + t) * a.q_stride + (size_t)g * DK + c] * a.q_scale : q_s[t * PK + c];
          const float k = L::CHANNEL ? a.k[(size_t)(first + t) * a.k_stride + (size_t)g * DK + c] : k_s[t * PK + c];
          const float w = L::CHANNEL ? w_s[t * PK + c] : small[t];
          if (MODE == CHUNK_WKV) {
            acc = fmaf(q, S[c], acc);
            bonus = fmaf(q * a.u[(size_t)h * DK + c], k, bonus);
          }
          S[c] = fmaf(w, S[c], k * v);
          if (MODE != CHUNK_WKV) acc = fmaf(q, S[c], acc);
        }
        if (MODE == CHUNK_WKV) acc = fmaf(bonus, v, acc);
        out[t * out_row + tid] = a.skip ? fmaf(skip, v, acc) : acc;
      }
#pragma unroll 1
      for (int c = 0; c < DK; ++c) local[(size_t)tid * DK + c] = S[c];
    }
    return;
  }

  {                                                        // o: a warp's 16 value channels, the first and last or the middle 16s of tokens
    const int m0 = warp >> 2, c0 = (warp & 3) * 16;        // rows of m0 and 3 - m0: five steps of 16 tokens either way
    float acc[2][2][4] = {};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      if (ks >= 4 - m0) break;
      FragB fb[2];
      load_b_columns(fb[0], v_s + ks * 16 * kPitchV + c0, kPitchV, lane);
      load_b_columns(fb[1], v_s + ks * 16 * kPitchV + c0 + 8, kPitchV, lane);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = i == 0 ? m0 : 3 - m0;
        if (ks <= m) {
          FragA fa;
          load_a_single(fa, a_s + m * kSub * kPitchA + ks * 16, kPitchA, lane);
          mma_split(acc[i][0], fa, fb[0]);
          mma_split(acc[i][1], fa, fb[1]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int t = (i == 0 ? m0 : 3 - m0) * kSub + half * 8 + (lane >> 2), c = c0 + j * 8 + 2 * (lane & 3);
          if (t < n) {
            float2 o = make_float2(acc[i][j][2 * half], acc[i][j][2 * half + 1]);
            if (a.skip) {
              o.x = fmaf(skip, v_s[t * kPitchV + c], o.x);
              o.y = fmaf(skip, v_s[t * kPitchV + c + 1], o.y);
            }
            *reinterpret_cast<float2*>(out + t * out_row + c) = o;
          }
        }
  }
  // what the stretch adds to the state: value channels as rows, 32 of them a warp, 16 key channels at a time
  const int v0 = (warp >> 2) * 32;
  for (int c0 = (warp & 3) * 16; c0 < DK; c0 += 64) {
    float acc[2][2][4] = {};
    float rest[2][4];                                      // CHANNEL: decays of the 16s behind the j-th
    if (L::CHANNEL) {
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        rest[x][3] = 1.0f;
#pragma unroll
        for (int j = 2; j >= 0; --j) rest[x][j] = rest[x][j + 1] * small[(j + 1) * DK + c0 + 8 * x + (lane >> 2)];
      }
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      FragA fa[2];
      load_a_columns(fa[0], v_s + ks * 16 * kPitchV + v0, kPitchV, lane);
      load_a_columns(fa[1], v_s + ks * 16 * kPitchV + v0 + 16, kPitchV, lane);
      float tail[4];                                       // decays from this lane's four tokens to the end
#pragma unroll
      for (int i = 0; i < 4; ++i) tail[i] = L::CHANNEL ? 1.0f : small[2 * kChunk + ks * 16 + (lane & 3) + 4 * i];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float* at = k_s + (ks * 16 + (lane & 3)) * PK + c0 + 8 * x + (lane >> 2);
        auto key = [&](int i) { return at[4 * i * PK] * (L::CHANNEL ? rest[x][ks] : tail[i]); };
        FragB fb;
        fb.v[0].set(key(0), key(2));
        fb.v[1].set(key(1), key(3));
        mma_split(acc[0][x], fa[0], fb);
        mma_split(acc[1][x], fa[1], fb);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        float* to = local + (size_t)(v0 + i * 16 + (lane >> 2)) * DK + c0 + 8 * x + 2 * (lane & 3);
        *reinterpret_cast<float2*>(to) = make_float2(acc[i][x][0], acc[i][x][1]);
        *reinterpret_cast<float2*>(to + 8 * DK) = make_float2(acc[i][x][2], acc[i][x][3]);
      }
  }
}

// grid (requests, heads, pieces of a state): four key channels of a value channel a thread.  The reads of eight stretches are
// on their way together; only the multiply-adds are in sequence.
template <bool CHANNEL, int PER>
__global__ void __launch_bounds__(256) chunk_carry_kernel(const ChunkArgs a, int dk) {
  const int r = blockIdx.x, h = blockIdx.y, e = blockIdx.z * 256 + threadIdx.x;
  const int lo = a.cu_seqlens[r], span = a.cu_seqlens[r + 1] - lo, chunks = chunks_of(span, a.min_span, PER);
  if (chunks == 0) return;
  if (a.x != nullptr && h == 0 && blockIdx.z == 0) {                       // the step's last input row
    float* to = a.prev_state + (long long)a.req_slot[r] * a.state_slot_stride;
    for (int i = threadIdx.x; i < a.C; i += 256) to[i] = a.x[(size_t)(lo + span - 1) * a.C + i];
  }
  if (e >= a.dv * (dk / 4)) return;
  const int v = e / (dk / 4), c = e % (dk / 4) * 4;
  float* st = a.state + (long long)a.req_slot[r] * a.state_slot_stride + (size_t)h * a.dv * dk;
  float4 S;
  if (a.key_rows) S = make_float4(st[(size_t)c * a.dv + v], st[(size_t)(c + 1) * a.dv + v], st[(size_t)(c + 2) * a.dv + v], st[(size_t)(c + 3) * a.dv + v]);
  else S = make_float4(st[(size_t)v * dk + c], st[(size_t)v * dk + c + 1], st[(size_t)v * dk + c + 2], st[(size_t)v * dk + c + 3]);
  const size_t base = (size_t)chunks_before(a.cu_seqlens, a.min_span, r, PER) * a.heads + h;
  constexpr int U = 8;
  for (int c0 = 0; c0 < chunks; c0 += U) {
    float4 add[U], w[U];
    float rest[U];                                         // what the one decay of a head lacks
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const size_t item = base + (size_t)min(c0 + i, chunks - 1) * a.heads;
      add[i] = *reinterpret_cast<const float4*>(a.local + (item * a.dv + v) * dk + c);
      if (CHANNEL) w[i] = *reinterpret_cast<const float4*>(a.total + item * dk + c);
      else {
        const float2 f = *reinterpret_cast<const float2*>(a.total + 2 * item);
        w[i] = make_float4(f.x, f.x, f.x, f.x);
        rest[i] = f.y;
      }
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (c0 + i < chunks) {
        *reinterpret_cast<float4*>(a.local + ((base + (size_t)(c0 + i) * a.heads) * a.dv + v) * dk + c) = S;
        if (!CHANNEL) {
          auto with_rest = [&](float s, float a) { return isfinite(s) ? fmaf(rest[i], s, a) : a; };
          add[i].x = with_rest(S.x, add[i].x);
          add[i].y = with_rest(S.y, add[i].y);
          add[i].z = with_rest(S.z, add[i].z);
          add[i].w = with_rest(S.w, add[i].w);
        }
        S.x = fmaf(w[i].x, S.x, add[i].x);
        S.y = fmaf(w[i].y, S.y, add[i].y);
        S.z = fmaf(w[i].z, S.z, add[i].z);
        S.w = fmaf(w[i].w, S.w, add[i].w);
      }
    }
  }
  const float s[4] = {S.x, S.y, S.z, S.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (a.key_rows) st[(size_t)(c + i) * a.dv + v] = s[i];
    else st[(size_t)v * dk + c + i] = s[i];
  }
}

// out += (queries times decays)^T state.  CHANNEL: the decays are in `reach` already; else its number scales a token's row.
template <int DK, bool CHANNEL>
__global__ void __launch_bounds__(256, 3) chunk_reach_kernel(const ChunkArgs a) {
  constexpr int PK = DK + 8;
  extern __shared__ __align__(16) float smem[];
  float *q_s = smem, *s_s = smem + kChunk * PK;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, z = blockIdx.z, g = h / (a.heads / a.groups), dv = a.dv;
  int first, n;
  if (!chunk_of(a.cu_seqlens, a.requests, a.min_span, blockIdx.x, first, n)) return;
  const float* state = a.local + (((size_t)blockIdx.x * a.heads + h) * dv + z * 64) * DK;
  bool bad = false;
#pragma unroll
  for (int e = tid; e < kChunk * DK / 4; e += 256) {
    const int t = e / (DK / 4), c = e % (DK / 4) * 4;
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < n) {
      if (CHANNEL) {
        q = *reinterpret_cast<const float4*>(a.reach + ((size_t)(first + t) * a.heads + h) * DK + c);
      } else {
        q = *reinterpret_cast<const float4*>(a.q + (size_t)(first + t) * a.q_stride + (size_t)g * DK + c);
        const float f = a.q_scale;
        q.x *= f; q.y *= f; q.z *= f; q.w *= f;
      }
    }
    const float4 s = *reinterpret_cast<const float4*>(state + (size_t)t * DK + c);        // row t: a value channel
    bad = bad || !splits(q) || !splits(s);
    *reinterpret_cast<float4*>(q_s + t * PK + c) = q;
    *reinterpret_cast<float4*>(s_s + t * PK + c) = s;
  }
  bad = __syncthreads_or(bad);
  float* out = a.out + (size_t)first * a.heads * dv + (size_t)h * dv + z * 64;
  const size_t out_row = (size_t)a.heads * dv;
  if (bad) {
    for (int e = tid; e < n * 64; e += 256) {
      const int t = e >> 6, c = e & 63;
      const float f = CHANNEL ? 1.0f : a.reach[(size_t)(first + t) * a.heads + h];
      float acc = 0.0f;
      for (int i = 0; i < DK; ++i) acc = fmaf(q_s[t * PK + i] * f, s_s[c * PK + i], acc);
      out[t * out_row + c] += acc;
    }
    return;
  }
  const int t0 = (warp >> 2) * 32, c0 = (warp & 3) * 16;   // a warp's 32 tokens and 16 value channels
  float2 before[2][2][2];                                  // the outputs so far: on their way under the products
  float scale[2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int t = min(t0 + i * 16 + half * 8 + (lane >> 2), n - 1);
      scale[i][half] = CHANNEL ? 1.0f : a.reach[(size_t)(first + t) * a.heads + h];
#pragma unroll
      for (int j = 0; j < 2; ++j) before[i][half][j] = *reinterpret_cast<const float2*>(out + t * out_row + c0 + j * 8 + 2 * (lane & 3));
    }
  float acc[2][2][4] = {};
#pragma unroll 2
  for (int kk = 0; kk < DK; kk += 16) {
    FragB fb[2];
    load_b_rows(fb[0], s_s + c0 * PK + kk, PK, lane);
    load_b_rows(fb[1], s_s + (c0 + 8) * PK + kk, PK, lane);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      FragA fa;
      load_a_rows(fa, q_s + (t0 + i * 16) * PK + kk, PK, lane);
      mma_split(acc[i][0], fa, fb[0]);
      mma_split(acc[i][1], fa, fb[1]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int t = t0 + i * 16 + half * 8 + (lane >> 2);
      if (t < n) {
        const float f = scale[i][half];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 o = before[i][half][j];
          *reinterpret_cast<float2*>(out + t * out_row + c0 + j * 8 + 2 * (lane & 3)) =
              make_float2(fmaf(f, acc[i][j][2 * half], o.x), fmaf(f, acc[i][j][2 * half + 1], o.y));
        }
      }
    }
}

template <int DK, int MODE>
static int launch_chunks(const ChunkArgs& a, int chunks, cudaStream_t stream) {
  using L = ChunkLayout<DK, MODE>;
  auto local = chunk_local_kernel<DK, MODE>;
  auto reach = chunk_reach_kernel<DK, L::CHANNEL>;
  const size_t reach_bytes = (size_t)2 * kChunk * (DK + 8) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(local, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES);
  if (e == cudaSuccess && reach_bytes > 48 * 1024) e = cudaFuncSetAttribute(reach, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)reach_bytes);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid(chunks, a.heads, a.dv / 64);
  local<<<grid, 256, L::BYTES, stream>>>(a);
  IFX_CHECK_LAUNCH();
  chunk_carry_kernel<L::CHANNEL, kChunk><<<dim3(a.requests, a.heads, (a.dv * (DK / 4) + 255) / 256), 256, 0, stream>>>(a, DK);
  IFX_CHECK_LAUNCH();
  reach<<<grid, 256, reach_bytes, stream>>>(a);
  IFX_CHECK_LAUNCH();
  return 0;
}

// The states in front of every stretch, for chunk_tcgen05.cu's stretches.  (Their size is a constant of the kernel: every block counts the
// stretches of the requests in front of its own, and with a division by a variable 32 requests took 3 to 5 % longer.)
int launch_chunk_carry(const ChunkArgs& a, int dk, cudaStream_t stream) {
  chunk_carry_kernel<false, 128><<<dim3(a.requests, a.heads, (a.dv * (dk / 4) + 255) / 256), 256, 0, stream>>>(a, dk);
  IFX_CHECK_LAUNCH();
  return 0;
}
int launch_chunks_of_128(const ChunkArgs& a, int dk, int mode, int chunks, int* error_flag, cudaStream_t stream);      // chunk_tcgen05.cu
bool chunks_of_128_take(int mode, int dk, int dv);

static int run_chunks(const ChunkArgs& a, int dk, int mode, int chunks, cudaStream_t stream) {
  if (dk == 64) {
    if (mode == CHUNK_CHANNEL) return launch_chunks<64, CHUNK_CHANNEL>(a, chunks, stream);
    if (mode == CHUNK_STEP) return launch_chunks<64, CHUNK_STEP>(a, chunks, stream);
    if (mode == CHUNK_CONSTANT) return launch_chunks<64, CHUNK_CONSTANT>(a, chunks, stream);
    return launch_chunks<64, CHUNK_WKV>(a, chunks, stream);
  }
  if (mode == CHUNK_CHANNEL) return launch_chunks<128, CHUNK_CHANNEL>(a, chunks, stream);
  if (mode == CHUNK_STEP) return launch_chunks<128, CHUNK_STEP>(a, chunks, stream);
  if (mode == CHUNK_CONSTANT) return launch_chunks<128, CHUNK_CONSTANT>(a, chunks, stream);
  return launch_chunks<128, CHUNK_WKV>(a, chunks, stream);
}

// The last of the three alone, for delta_chunks.cu: heads of 64 x 64, `reach` [T, heads 64] and the states as chunk_carry leaves them.
int launch_chunk_reach_64(const float* reach, const float* local, float* out, const int* cu_seqlens, int requests, int min_span, int heads,
                          int chunks, cudaStream_t stream) {
  ChunkArgs a = {};
  a.reach = const_cast<float*>(reach);
  a.local = const_cast<float*>(local);
  a.out = out;
  a.cu_seqlens = cu_seqlens;
  a.requests = requests;
  a.min_span = min_span;
  a.heads = a.groups = heads;
  a.dv = 64;
  chunk_reach_kernel<64, true><<<dim3(chunks, heads, 1), 256, 2 * kChunk * (64 + 8) * sizeof(float), stream>>>(a);
  IFX_CHECK_LAUNCH();
  return 0;
}

static bool rows_fit(const void* p, long long stride) { return stride % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace ifx

using namespace ifx;

extern "C" {

// 1 if the kernels take these sizes and this many requests (the stretches are found by walking the requests).
int ifx_chunk_scan_supports(int requests, int heads, int dk, int dv) {
  return requests > 0 && requests <= 64 && heads > 0 && heads <= 65535 && (dk == 64 || dk == 128) && dv > 0 && dv % 64 == 0 && dv / 64 <= 65535;
}

// Floats of scratch.  per_channel: a decay per key channel (mode 0 and wkv).  min_span here and below: spans with fewer tokens are
// not touched (1: none are left out).
long long ifx_chunk_scan_scratch_floats(int num_tokens, int requests, int min_span, int heads, int dk, int dv, int per_channel) {
  const long long chunks = chunks_at_most(num_tokens, requests, min_span);
  const long long total = ((per_channel ? chunks * heads * dk : 2 * chunks * heads) + 3) / 4 * 4;
  return chunks * heads * dv * dk + total + (per_channel ? (long long)num_tokens * heads * dk : (long long)num_tokens * heads);
}

// Whether a decay per head goes by stretches of 128 tokens (chunk_tcgen05.cu) where they take the sizes: when the blocks of the stretches of
// 64 would not all have an SM of their own.  us, by 64 and by 128: 12 heads of 128 x 128, one span of 300 tokens 30 / 35, 512 43 / 36,
// 2,048 119 / 64; 12 of 64 x 128 22 / 28, 29 / 29, 69 / 49; 24 of 128 x 64 31 / 32, 44 / 33, 115 / 67; 28 of 128 x 128, 128 tokens 44 / 36; but 56
// of 128 x 64, 256 tokens 45.5 / 47.0.
int ifx_chunk_scan_takes_128(int num_tokens, int num_requests, int min_span, int heads, int dv) {
  return (long long)chunks_at_most(num_tokens, num_requests, min_span) * heads * (dv / 64) > 148;
}

// As ifx_decay_scan_rate (decay_scan.cu), with scratch as above; every row on a 16-byte boundary (IFX_E_ALIGN otherwise).  stretch: 64 or 128
// tokens (where those take the sizes), or 0 for what ifx_chunk_scan_takes_128 says.
int ifx_chunk_decay_scan(const float* q, long long q_stride, const float* k, long long k_stride, const float* v, long long v_stride,
                         const float* raw, long long raw_stride, float* state, long long state_slot_stride, const int* req_slot,
                         const int* cu_seqlens, float* out, const float* step_bias, const float* log_rate, const float* skip,
                         int num_requests, int num_tokens, int min_span, int heads, int groups, int dk, int dv, int mode, float tau,
                         float q_scale, float* scratch, const float* rate, int stretch, int* error_flag, cudaStream_t stream) {
  if (num_requests <= 0 || num_tokens <= 0 || num_tokens < min_span) return 0;
  if (!ifx_chunk_scan_supports(num_requests, heads, dk, dv) || groups <= 0 || heads % groups || mode < 0 || mode > 2 || scratch == nullptr)
    return IFX_E_BADARG;
  if ((mode == 0 && !(tau > 0.0f)) || (mode == 1 && (step_bias == nullptr || log_rate == nullptr)) || (mode == 2 && rate == nullptr))
    return IFX_E_BADARG;
  if (!rows_fit(q, q_stride) || !rows_fit(k, k_stride) || !rows_fit(v, v_stride) || (mode == 0 && !rows_fit(raw, raw_stride)) ||
      !rows_fit(scratch, 0) || !rows_fit(out, 0))
    return IFX_E_ALIGN;
  const int per = (stretch == 128 || (stretch == 0 && ifx_chunk_scan_takes_128(num_tokens, num_requests, min_span, heads, dv))) &&
                          chunks_of_128_take(mode, dk, dv) && error_flag != nullptr ? 128 : kChunk;
  const int chunks = chunks_at_most(num_tokens, num_requests, min_span, per);
  ChunkArgs a = {};
  a.q = q; a.q_stride = q_stride; a.k = k; a.k_stride = k_stride; a.v = v; a.v_stride = v_stride; a.raw = raw; a.raw_stride = raw_stride;
  a.state = state; a.state_slot_stride = state_slot_stride; a.req_slot = req_slot; a.cu_seqlens = cu_seqlens; a.out = out;
  a.step_bias = step_bias; a.log_rate = log_rate; a.skip = skip; a.rate = rate;
  a.requests = num_requests; a.min_span = min_span; a.heads = heads; a.groups = groups; a.dv = dv;
  a.inv_tau = mode == 0 ? 1.0f / tau : 0.0f;
  a.q_scale = q_scale;
  a.local = scratch;
  a.total = scratch + (size_t)chunks * heads * dv * dk;
  a.reach = a.total + ((mode == 0 ? (size_t)chunks * heads * dk : (size_t)2 * chunks * heads) + 3) / 4 * 4;
  if (per == 128) return launch_chunks_of_128(a, dk, mode, chunks, error_flag, stream);
  return run_chunks(a, dk, mode, chunks, stream);
}

// As the recurrence of ifx_wkv_scan (wkv.cu) without the norm and gate behind it: out [T, heads dim] float32.
int ifx_chunk_wkv_scan(const float* r, const float* k, const float* v, const float* w_raw, const float* w0, const float* u,
                       float* s_state, float* prev_state, long long slot_stride, const float* x, int C, const int* cu_seqlens,
                       const int* req_slot, float* out, int num_requests, int num_tokens, int min_span, int heads, int dim, int ld,
                       int ld_w, float* scratch, cudaStream_t stream) {
  if (num_requests <= 0 || num_tokens <= 0 || num_tokens < min_span) return 0;
  if (!ifx_chunk_scan_supports(num_requests, heads, dim, dim) || scratch == nullptr) return IFX_E_BADARG;
  if (!rows_fit(r, ld) || !rows_fit(k, ld) || !rows_fit(v, ld) || !rows_fit(w_raw, ld_w) || !rows_fit(w0, 0) || !rows_fit(u, 0) ||
      !rows_fit(scratch, 0) || !rows_fit(out, 0))
    return IFX_E_ALIGN;
  const int chunks = chunks_at_most(num_tokens, num_requests, min_span);
  ChunkArgs a = {};
  a.q = r; a.q_stride = ld; a.k = k; a.k_stride = ld; a.v = v; a.v_stride = ld; a.raw = w_raw; a.raw_stride = ld_w;
  a.state = s_state; a.state_slot_stride = slot_stride; a.req_slot = req_slot; a.cu_seqlens = cu_seqlens; a.out = out;
  a.w0 = w0; a.u = u; a.x = x; a.prev_state = prev_state; a.C = C;
  a.requests = num_requests; a.min_span = min_span; a.heads = heads; a.groups = heads; a.dv = dim;
  a.q_scale = 1.0f;
  a.key_rows = 1;
  a.local = scratch;
  a.total = scratch + (size_t)chunks * heads * dim * dim;
  a.reach = a.total + (size_t)chunks * heads * dim;
  return run_chunks(a, dim, CHUNK_WKV, chunks, stream);
}

}  // extern "C"
