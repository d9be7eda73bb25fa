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
// a unit lower triangular system, solved for the columns of [N V | U] so that everything is linear in S_0.  Four kernels:
//
//   delta_local   per stretch and head: outputs without S_0, the queries that meet S_0, the matrix that carries S_0 on, what is added
//   delta_carry   the states in front of every stretch, one small product a stretch, 16 value channels a block
//   chunk_reach   (chunk_scan.cu) adds what S_0 brings to the outputs
//   delta_finish  (delta_rule.cu) norm and gate
//
// A decay lies between 0.545 and 1, so products over half a stretch and their reciprocals stay below 3e8: G_t / G_s is taken as
// a product on the one side and a reciprocal on the other, both counted from the middle of the stretch.  Products run on the tensor
// cores with split operands (chunk_scan.cuh); the triangular system goes by blocks of 16 rows, substituted in the blocks.
//
// A stretch that holds a number that is not finite, or in which one comes up that a scan would not have formed, is walked token by
// token.  The order of the sums depends on where a span is cut into steps, so the float32 run keeps the scan.
//
// Bound: delta_local, one block of 16 warps an SM (128 KB): twenty barriers and the chain split -> product -> sum between them (issue
// slots 44 % busy, tensor pipe 29 %).  2,048 tokens of 24 heads: delta_rule.cu's three kernels 658 us, these 303.
// Error of the state against 64 bits (2-norm, scan and this, 2,048 tokens): parameters where trained models have them 5.2e-7 and
// 4.6e-7, decays near one 1.76e-6 and 1.70e-6, random ones 0.95e-7 and 1.00e-7.  (With operands of 22 bits 241 us, 1.4e-7 in the last
// case, and 1.0e-6 in place of the scan's 4.6e-7 where 130 keys are nearly the same.)
#include "chunk_scan.cuh"

namespace ifx {

constexpr int kDcThreads = 512, kDcD = 64, kDcP = kPitchV;
constexpr float kDcFloor = 0.6065306597126334f;            // exp(-1/2)

struct DeltaChunkArgs {
  const float* proj; int ld;                                // r, k, v, g, a in column blocks of heads * 64
  const float* w_raw; const float* w0; const float* a_bias;
  float* state; long long state_slot_stride; const int* req_slot; const int* cu_seqlens;
  float* out;                                               // [T, heads 64]
  int requests, min_span, heads;                            // shorter spans are left to delta_scan
  float *local, *trans, *reach;                             // [stretches, heads, v, k], [stretches, heads, k, k], [T, heads 64]
};

struct DeltaChunkLayout {
  static constexpr int TILE = kChunk * kDcP;
  static constexpr int R = 0, U = TILE, K = 2 * TILE, E = 3 * TILE, V = 4 * TILE, X = 5 * TILE, A = 6 * TILE, MID = A + kChunk * kPitchA,
                       END = MID + kDcD, FLOATS = END + kDcD;
  static constexpr size_t BYTES = (size_t)FLOATS * sizeof(float);
};

// acc = rows . columns^T of two tiles whose inner size runs along the rows; 16 rows x 16 columns a warp.
__device__ __forceinline__ void dc_pairs(float (&acc)[2][4], const float* x, const float* y, int lane) {
#pragma unroll
  for (int kk = 0; kk < kDcD; kk += 16) {
    FragA fa;
    FragB fb;
    load_a_rows(fa, x + kk, kDcP, lane);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      load_b_rows(fb, y + j * 8 * kDcP + kk, kDcP, lane);
      mma_split(acc[j], fa, fb);
    }
  }
}
// acc += the first `steps` sixteens of a row of the matrix times the rows of a tile.
__device__ __forceinline__ void dc_times(float (&acc)[2][4], const float* a, const float* tile, int steps, int lane) {
  for (int ks = 0; ks < steps; ++ks) {
    FragA fa;
    FragB fb;
    load_a_single(fa, a + ks * 16, kPitchA, lane);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      load_b_columns(fb, tile + ks * 16 * kDcP + j * 8, kDcP, lane);
      mma_split(acc[j], fa, fb);
    }
  }
}
// acc = columns of one tile . columns of another, over the tokens.
__device__ __forceinline__ void dc_over_tokens(float (&acc)[2][4], const float* x, const float* y, int lane) {
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    FragA fa;
    FragB fb;
    load_a_columns(fa, x + ks * 16 * kDcP, kDcP, lane);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      load_b_columns(fb, y + ks * 16 * kDcP + j * 8, kDcP, lane);
      mma_split(acc[j], fa, fb);
    }
  }
}
__device__ __forceinline__ float dc_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

__global__ void __launch_bounds__(kDcThreads, 1) delta_local_kernel(const DeltaChunkArgs a) {
  using L = DeltaChunkLayout;
  extern __shared__ __align__(16) float smem[];
  float *r_s = smem + L::R, *u_s = smem + L::U, *k_s = smem + L::K, *e_s = smem + L::E, *v_s = smem + L::V, *x_s = smem + L::X,
        *a_s = smem + L::A, *mid = smem + L::MID, *end = smem + L::END;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, HD = a.heads * kDcD;
  int first, n;
  if (!chunk_of(a.cu_seqlens, a.requests, a.min_span, blockIdx.x, first, n)) return;
  const size_t item = (size_t)blockIdx.x * a.heads + h;

  // ---------------------------------------------------------- rows: queries, keys, values, how much is erased, unit keys, decays
  auto load = [&]() {
    bool bad = false;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int t = half * 32 + (tid >> 4), c = (tid & 15) * 4;             // sixteen neighbouring lanes a token
      float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f), k = r, v = r, e = r, w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
      if (t < n) {
        const float* row = a.proj + (size_t)(first + t) * a.ld + h * kDcD + c;
        r = *reinterpret_cast<const float4*>(row);
        k = *reinterpret_cast<const float4*>(row + HD);
        v = *reinterpret_cast<const float4*>(row + 2 * HD);
        e = *reinterpret_cast<const float4*>(row + 4 * HD);
        w = *reinterpret_cast<const float4*>(a.w_raw + (size_t)(first + t) * HD + h * kDcD + c);
        const float4 b = *reinterpret_cast<const float4*>(a.a_bias + h * kDcD + c), w0 = *reinterpret_cast<const float4*>(a.w0 + h * kDcD + c);
        e.x = dc_sigmoid(e.x + b.x); e.y = dc_sigmoid(e.y + b.y); e.z = dc_sigmoid(e.z + b.z); e.w = dc_sigmoid(e.w + b.w);
        w.x = expf(-kDcFloor * dc_sigmoid(w.x + w0.x)); w.y = expf(-kDcFloor * dc_sigmoid(w.y + w0.y));
        w.z = expf(-kDcFloor * dc_sigmoid(w.z + w0.z)); w.w = expf(-kDcFloor * dc_sigmoid(w.w + w0.w));
      }
      float ss = fmaf(k.x, k.x, fmaf(k.y, k.y, fmaf(k.z, k.z, k.w * k.w)));
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float inv = 1.0f / sqrtf(ss + 1e-6f);
      const float4 u = make_float4(k.x * inv, k.y * inv, k.z * inv, k.w * inv);
      e.x *= u.x; e.y *= u.y; e.z *= u.z; e.w *= u.w;
      bad = bad || !splits(r) || !splits(k) || !splits(v) || !splits(e) || !splits(w) || !isfinite(ss);
      *reinterpret_cast<float4*>(r_s + t * kDcP + c) = r;
      *reinterpret_cast<float4*>(k_s + t * kDcP + c) = k;
      *reinterpret_cast<float4*>(v_s + t * kDcP + c) = v;
      *reinterpret_cast<float4*>(e_s + t * kDcP + c) = e;
      *reinterpret_cast<float4*>(u_s + t * kDcP + c) = u;
      *reinterpret_cast<float4*>(a_s + t * kPitchA + c) = w;
    }
    return bad;
  };
  bool bad = __syncthreads_or(load());
  float* out = a.out + (size_t)first * HD + h * kDcD;
  float* reach = a.reach + (size_t)first * HD + h * kDcD;
  float *local = a.local + item * kDcD * kDcD, *trans = a.trans + item * kDcD * kDcD;

  auto walk = [&]() {                                      // token by token: 64 columns of values, 64 of the unit matrix
    if (tid < 2 * kDcD) {
      const bool unit = tid >= kDcD;
      const int j = tid & (kDcD - 1);
      float S[kDcD];                                       // in local memory: this path is for correctness
#pragma unroll 1
      for (int i = 0; i < kDcD; ++i) S[i] = unit && i == j ? 1.0f : 0.0f;
#pragma unroll 1
      for (int t = 0; t < n; ++t) {
        float x = 0.0f, kept = 0.0f, c1 = 0.0f, c2 = 0.0f;  // the output from the state in front of the token, as delta_scan_kernel takes it
        const float v = unit ? 0.0f : v_s[t * kDcP + j];
#pragma unroll 1
        for (int i = 0; i < kDcD; ++i) {
          const float r = r_s[t * kDcP + i];
          x = fmaf(u_s[t * kDcP + i], S[i], x);
          kept = fmaf(r * a_s[t * kPitchA + i], S[i], kept);
          c1 = fmaf(r, e_s[t * kDcP + i], c1);
          c2 = fmaf(r, k_s[t * kDcP + i], c2);
        }
#pragma unroll 1
        for (int i = 0; i < kDcD; ++i) {
          const float w = a_s[t * kPitchA + i] * S[i];
          S[i] = fmaf(-e_s[t * kDcP + i], x, unit ? w : fmaf(k_s[t * kDcP + i], v, w));
        }
        const float o = fmaf(-c1, x, unit ? kept : fmaf(c2, v, kept));
        (unit ? reach : out)[(size_t)t * HD + j] = o;
      }
#pragma unroll 1
      for (int i = 0; i < kDcD; ++i) (unit ? trans[i * kDcD + j] : local[j * kDcD + i]) = S[i];
    }
  };
  if (bad) {
    walk();
    return;
  }

  // ---------------------------------------------------------- decays from the middle: x_s holds G_t / G_31 for t > 31, its reciprocal up to there
  if (tid < 2 * kDcD) {
    const int c = tid & (kDcD - 1);
    Product p;
    if (tid < kDcD) {
      x_s[31 * kDcP + c] = 1.0f;
#pragma unroll 8
      for (int t = 30; t >= 0; --t) {
        p.times(a_s[(t + 1) * kPitchA + c]);
        x_s[t * kDcP + c] = p.value();
      }
      p.times(a_s[c]);
      mid[c] = p.value();                                  // from the stretch's beginning to the middle
    } else {
#pragma unroll 8
      for (int t = 32; t < kChunk; ++t) {
        p.times(a_s[t * kPitchA + c]);
        x_s[t * kDcP + c] = p.value();
      }
      end[c] = p.value();
    }
  }
  __syncthreads();
  uint32_t largest = 0;                                    // of what is made here to be split
  auto note = [&](float x) { largest = max(largest, magnitude(x)); };
#pragma unroll
  for (int e8 = 0; e8 < kChunk * kDcD / kDcThreads; ++e8) {
    const int e = e8 * kDcThreads + tid, t = e >> 6, c = e & 63;
    const float p = x_s[t * kDcP + c], q = 1.0f / p, f = t > 31 ? p : q, back = t > 31 ? q : p;
    const float before = t == 0 ? 1.0f / mid[c] : (t > 32 ? x_s[(t - 1) * kDcP + c] : 1.0f / x_s[(t - 1) * kDcP + c]);
    r_s[t * kDcP + c] *= f;
    u_s[t * kDcP + c] *= before;
    k_s[t * kDcP + c] *= back;
    e_s[t * kDcP + c] *= back;
    note(r_s[t * kDcP + c]);
    note(u_s[t * kDcP + c]);
    note(k_s[t * kDcP + c]);
    note(e_s[t * kDcP + c]);
  }
  __syncthreads();

  const int wm = warp >> 2, wn = warp & 3, steps = wm + 1;          // this warp's 16 rows and 16 columns
  const int tr = wm * 16 + (lane >> 2), tc = wn * 16 + 2 * (lane & 3);    // its first numbers: rows tr and tr + 8, columns tc + 8 j, + 1
  auto lower = [&](const float* rows, const float* cols, bool strict) {   // a_s = the lower triangle of rows . cols^T
    if (wn <= wm) {
      float acc[2][4] = {};
      dc_pairs(acc, rows + wm * 16 * kDcP, cols + wn * 16 * kDcP, lane);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = tr + (i >> 1) * 8, s = tc + j * 8 + (i & 1);
          const float x = (strict ? s < t : s <= t) ? acc[j][i] : 0.0f;
          a_s[t * kPitchA + s] = x;
          note(x);
        }
    }
  };
  lower(u_s, k_s, true);                                   // N
  __syncthreads();
  {
    float acc[2][4] = {};
    dc_times(acc, a_s + wm * 16 * kPitchA, v_s + wn * 16, steps, lane);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) x_s[(tr + (i >> 1) * 8) * kDcP + tc + j * 8 + (i & 1)] = acc[j][i];
  }
  __syncthreads();
  lower(r_s, k_s, false);                                  // A
  __syncthreads();
  float o[2][4] = {};
  dc_times(o, a_s + wm * 16 * kPitchA, v_s + wn * 16, steps, lane);
  __syncthreads();
  lower(u_s, e_s, true);                                   // M
  __syncthreads();
  for (int e = tid; e < kChunk * kDcD; e += kDcThreads) u_s[(e >> 6) * kDcP + (e & 63)] *= mid[e & 63];     // U, counted from the beginning
  __syncthreads();
  for (int i = 0; i < 4; ++i) {                            // [x_s | u_s] <- (1 + M)^-1 [x_s | u_s], 16 rows at a time
    if (tid < 2 * kDcD) {
      float* col = (tid < kDcD ? x_s : u_s) + i * 16 * kDcP + (tid & (kDcD - 1));
      const float* m = a_s + i * 16 * kPitchA + i * 16;
      float x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r] = col[r * kDcP];
      note(x[0]);
#pragma unroll
      for (int r = 1; r < 16; ++r) {
#pragma unroll
        for (int q = 0; q < r; ++q) x[r] = fmaf(-m[r * kPitchA + q], x[q], x[r]);
        col[r * kDcP] = x[r];
        note(x[r]);
      }
    }
    __syncthreads();
    for (int task = warp; task < (3 - i) * 8; task += 16) {               // what these rows take off the ones below
      const int j = i + 1 + (task >> 3), c = (task & 7) * 16;
      float* tile = (c < kDcD ? x_s : u_s) + (c & (kDcD - 1));
      float acc[2][4] = {};
      dc_times(acc, a_s + j * 16 * kPitchA + i * 16, tile + i * 16 * kDcP, 1, lane);
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          tile[(j * 16 + (lane >> 2) + (q >> 1) * 8) * kDcP + x * 8 + 2 * (lane & 3) + (q & 1)] -= acc[x][q];
    }
    __syncthreads();
  }
  lower(r_s, e_s, false);                                  // B
  if (__syncthreads_or(largest >= kSplitLimit)) {
    load();
    __syncthreads();
    walk();
    return;
  }
  {
    float bx[2][4] = {}, bu[2][4] = {};
    dc_times(bx, a_s + wm * 16 * kPitchA, x_s + wn * 16, steps, lane);
    dc_times(bu, a_s + wm * 16 * kPitchA, u_s + wn * 16, steps, lane);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = tr + half * 8, c = tc + j * 8;
        if (t < n) {
          *reinterpret_cast<float2*>(out + (size_t)t * HD + c) = make_float2(o[j][2 * half] - bx[j][2 * half], o[j][2 * half + 1] - bx[j][2 * half + 1]);
          *reinterpret_cast<float2*>(reach + (size_t)t * HD + c) =
              make_float2(fmaf(r_s[t * kDcP + c], mid[c], -bu[j][2 * half]), fmaf(r_s[t * kDcP + c + 1], mid[c + 1], -bu[j][2 * half + 1]));
        }
      }
  }
  {
    float kv[2][4] = {}, ex[2][4] = {}, eu[2][4] = {};
    dc_over_tokens(kv, v_s + wm * 16, k_s + wn * 16, lane);               // [v, k]
    dc_over_tokens(ex, x_s + wm * 16, e_s + wn * 16, lane);               // [v, k]
    dc_over_tokens(eu, e_s + wm * 16, u_s + wn * 16, lane);               // [k, k]
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = tr + half * 8, c = tc + j * 8;
        *reinterpret_cast<float2*>(local + row * kDcD + c) =
            make_float2((kv[j][2 * half] - ex[j][2 * half]) * end[c], (kv[j][2 * half + 1] - ex[j][2 * half + 1]) * end[c + 1]);
        const float f = end[row], g = f * mid[row];
        *reinterpret_cast<float2*>(trans + row * kDcD + c) =
            make_float2((row == c ? g : 0.0f) - f * eu[j][2 * half], (row == c + 1 ? g : 0.0f) - f * eu[j][2 * half + 1]);
      }
  }
}

// grid (requests, heads, 4): 16 value channels of a head along a request's stretches.  The next stretch's matrices arrive by
// cp.async while this one's product runs; a warp makes 16 x 8 numbers of it.
constexpr int kCarryThreads = 256;
constexpr int kCarryTrans = kDcD * kDcP, kCarryState = 16 * kDcP;

__global__ void __launch_bounds__(kCarryThreads) delta_carry_kernel(const DeltaChunkArgs a) {
  extern __shared__ __align__(16) float smem[];
  float* p_s = smem;                                       // [2][64][72]: the matrices
  float* l_s = p_s + 2 * kCarryTrans;                      // [2][16][72]: what is added
  float* s_s = l_s + 2 * kCarryState;                      // [16][72]: the state, a value channel a row
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * 16;
  const int chunks = chunks_of(a.cu_seqlens[r + 1] - a.cu_seqlens[r], a.min_span);
  if (chunks == 0) return;
  const size_t base = (size_t)chunks_before(a.cu_seqlens, a.min_span, r) * a.heads + h;
  float* st = a.state + (long long)a.req_slot[r] * a.state_slot_stride + (size_t)h * kDcD * kDcD;      // [k, v]
  bool bad = false;                                        // numbers of the state, the matrix that are not finite: split products would lose them
  for (int e = tid; e < 16 * kDcD; e += kCarryThreads) {
    const float v = st[(e >> 4) * kDcD + v0 + (e & 15)];
    bad = bad || !splits(v);
    s_s[(e & 15) * kDcP + (e >> 4)] = v;
  }
  auto copy = [](float* to, const float* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from) : "memory");
  };
  auto fetch = [&](int c) {
    const size_t item = base + (size_t)c * a.heads;
    float *p = p_s + (c & 1) * kCarryTrans, *l = l_s + (c & 1) * kCarryState;
    for (int e = tid; e < kDcD * 16; e += kCarryThreads) copy(p + (e >> 4) * kDcP + (e & 15) * 4, a.trans + item * kDcD * kDcD + e * 4);
    copy(l + (tid >> 4) * kDcP + (tid & 15) * 4, a.local + item * kDcD * kDcD + (size_t)v0 * kDcD + tid * 4);
  };
  fetch(0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  const int wm = warp >> 1, wn = warp & 1;                 // 16 key channels, 8 value channels
  for (int c = 0; c < chunks; ++c) {
    if (c + 1 < chunks) fetch(c + 1);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
    const float *p = p_s + (c & 1) * kCarryTrans, *l = l_s + (c & 1) * kCarryState;
    for (int e = tid; e < kDcD * 16; e += kCarryThreads)
      bad = bad || !splits(*reinterpret_cast<const float4*>(p + (e >> 4) * kDcP + (e & 15) * 4));
    bad = __syncthreads_or(bad);
    *reinterpret_cast<float4*>(a.local + (base + (size_t)c * a.heads) * kDcD * kDcD + (size_t)v0 * kDcD + tid * 4) =
        *reinterpret_cast<const float4*>(s_s + (tid >> 4) * kDcP + (tid & 15) * 4);       // the state in front of the stretch
    float acc[2][4] = {};
    const int k0 = wm * 16 + (lane >> 2), vc = wn * 8 + 2 * (lane & 3);
    if (bad) {
#pragma unroll 1
      for (int j = 0; j < kDcD; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[0][i] = fmaf(p[(k0 + (i >> 1) * 8) * kDcP + j], s_s[(vc + (i & 1)) * kDcP + j], acc[0][i]);
    } else {
#pragma unroll
      for (int kk = 0; kk < kDcD; kk += 16) {
        FragA fa;
        FragB fb;
        load_a_rows(fa, p + wm * 16 * kDcP + kk, kDcP, lane);
        load_b_rows(fb, s_s + wn * 8 * kDcP + kk, kDcP, lane);
        mma_split(acc[(kk >> 4) & 1], fa, fb);
      }
    }
    __syncthreads();                                       // the state has been read by all
    bad = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + (i >> 1) * 8, v = vc + (i & 1);
      const float x = acc[0][i] + acc[1][i] + l[v * kDcP + k];
      bad = bad || !splits(x);
      s_s[v * kDcP + k] = x;
    }
    __syncthreads();
  }
  for (int e = tid; e < 16 * kDcD; e += kCarryThreads) st[(e >> 4) * kDcD + v0 + (e & 15)] = s_s[(e & 15) * kDcP + (e >> 4)];
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
  return 2LL * chunks_at_most(num_tokens, requests, min_span) * heads * kDcD * kDcD + 2LL * num_tokens * heads * kDcD;
}

// As ifx_delta_rule_scan (delta_rule.cu) for heads of 64 channels, with scratch as above; rows on 16-byte boundaries.  Spans of
// fewer than min_span tokens go through delta_scan, with scan_scratch as ifx_delta_rule_scratch_floats says (null: there are none).
int ifx_delta_chunks_scan(const float* proj, int ld, const float* w_raw, const float* w0, const float* a_bias, const float* norm_w,
                          float eps, float* state, long long slot_stride, const int* cu_seqlens, const int* req_slot, float* scratch,
                          void* y, int num_requests, int num_tokens, int min_span, int heads, int dim, int out_dtype, float* scan_scratch,
                          cudaStream_t stream) {
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
  const size_t states = (size_t)chunks * heads * kDcD * kDcD, rows = (size_t)num_tokens * heads * kDcD;
  a.local = scratch;
  a.trans = a.local + states;
  a.reach = a.trans + states;
  a.out = a.reach + rows;
  const size_t carry_bytes = (size_t)(2 * kCarryTrans + 3 * kCarryState) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(delta_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DeltaChunkLayout::BYTES);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_carry_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)carry_bytes);
  if (e != cudaSuccess) return (int)e;
  if (scan_scratch != nullptr) {
    const int rc = launch_delta_scan(proj, ld, w_raw, w0, a_bias, state, slot_stride, cu_seqlens, req_slot, scan_scratch, a.out, num_requests,
                                     num_tokens, heads, dim, min_span - 1, stream);
    if (rc) return rc;
  }
  delta_local_kernel<<<dim3(chunks, heads), kDcThreads, DeltaChunkLayout::BYTES, stream>>>(a);
  IFX_CHECK_LAUNCH();
  delta_carry_kernel<<<dim3(num_requests, heads, 4), kCarryThreads, carry_bytes, stream>>>(a);
  IFX_CHECK_LAUNCH();
  const int rc = launch_chunk_reach_64(a.reach, a.local, a.out, cu_seqlens, num_requests, min_span, heads, chunks, stream);
  if (rc) return rc;
  return launch_delta_finish(a.out, proj, ld, norm_w, eps, y, num_tokens, heads, dim, out_dtype, stream);
}

}  // extern "C"
