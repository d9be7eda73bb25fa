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
//   delta_carry   the states in front of every stretch, one small product a stretch, 8 value channels a block
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
// Bound: delta_local, two blocks of 8 warps an SM (110 KB each: X in the values' place, decays in the matrix's): barriers and the chain
// split -> product -> sum between them (issue slots 49 % busy, tensor pipe 35 %; one block of 16 warps with a tile more 206 us, so
// 165).  2,048 tokens of 24 heads: delta_rule.cu's three kernels 658 us, these 232.
// Error of the state against 64 bits (2-norm, scan and this, 2,048 tokens): parameters where trained models have them 5.2e-7 and
// 4.6e-7, decays near one 1.76e-6 and 1.70e-6, random ones 0.95e-7 and 1.00e-7.  (With operands of 22 bits 241 us, 1.4e-7 in the last
// case, and 1.0e-6 in place of the scan's 4.6e-7 where 130 keys are nearly the same.)
#include "chunk_scan.cuh"

namespace ifx {

constexpr int kDcThreads = 256, kDcD = 64, kDcP = kPitchV;
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

struct DeltaChunkLayout {
  static constexpr int TILE = kChunk * kDcP;
  static constexpr int R = 0, U = TILE, K = 2 * TILE, E = 3 * TILE, V = 4 * TILE, A = 5 * TILE, MID = A + kChunk * kPitchA,
                       END = MID + kDcD, FLOATS = END + kDcD;
  static constexpr size_t BYTES = (size_t)FLOATS * sizeof(float);
};

// A warp makes 16 columns of two blocks of 16 rows: the first and the last, or the two in the middle.  Both halves of the warps then
// have the same share of what lies below a diagonal, and split a column operand once for both.
struct DcTile {
  int r0, r1, c;                                            // rows of the two blocks, columns
  __device__ __forceinline__ DcTile(int warp) : r0((warp >> 2) * 16), r1(48 - (warp >> 2) * 16), c((warp & 3) * 16) {}
  __device__ __forceinline__ int row(int b) const { return b ? r1 : r0; }
};
typedef float DcAcc[2][2][4];                               // block of rows, 8 columns, the product's own order

// acc = rows . columns^T of two tiles whose inner size runs along the rows, in the blocks on and below the diagonal.
__device__ __forceinline__ void dc_pairs(DcAcc& acc, const float* x, const float* y, const DcTile& w, int lane) {
  if (w.c > w.r1) return;
#pragma unroll 2
  for (int kk = 0; kk < kDcD; kk += 16) {
    FragA fa;
    FragB fb[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) load_b_rows(fb[j], y + (w.c + j * 8) * kDcP + kk, kDcP, lane);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      if (w.c > w.row(b)) continue;
      load_a_rows(fa, x + w.row(b) * kDcP + kk, kDcP, lane);
#pragma unroll
      for (int j = 0; j < 2; ++j) mma_split(acc[b][j], fa, fb[j]);
    }
  }
}
// acc += the lower triangle of a matrix times the rows of a tile.
__device__ __forceinline__ void dc_times(DcAcc& acc, const float* m, const float* tile, const DcTile& w, int lane) {
  for (int s = 0; s <= w.r1; s += 16) {
    FragA fa;
    FragB fb[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) load_b_columns(fb[j], tile + s * kDcP + w.c + j * 8, kDcP, lane);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      if (s > w.row(b)) continue;
      load_a_single(fa, m + w.row(b) * kPitchA + s, kPitchA, lane);
#pragma unroll
      for (int j = 0; j < 2; ++j) mma_split(acc[b][j], fa, fb[j]);
    }
  }
}
// acc = columns of one tile . columns of another, over the tokens.
__device__ __forceinline__ void dc_over_tokens(DcAcc& acc, const float* x, const float* y, const DcTile& w, int lane) {
#pragma unroll 2
  for (int s = 0; s < kChunk; s += 16) {
    FragA fa;
    FragB fb[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) load_b_columns(fb[j], y + s * kDcP + w.c + j * 8, kDcP, lane);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      load_a_columns(fa, x + s * kDcP + w.row(b), kDcP, lane);
#pragma unroll
      for (int j = 0; j < 2; ++j) mma_split(acc[b][j], fa, fb[j]);
    }
  }
}
__device__ __forceinline__ float dc_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

__global__ void __launch_bounds__(kDcThreads, 2) delta_local_kernel(const DeltaChunkArgs a) {
  using L = DeltaChunkLayout;
  extern __shared__ __align__(16) float smem[];
  float *r_s = smem + L::R, *u_s = smem + L::U, *k_s = smem + L::K, *e_s = smem + L::E, *v_s = smem + L::V,
        *a_s = smem + L::A, *mid = smem + L::MID, *end = smem + L::END;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, HD = a.heads * kDcD;
  int first, n;
  if (!chunk_of(a.cu_seqlens, a.requests, a.min_span, blockIdx.x, first, n)) return;
  const size_t item = (size_t)blockIdx.x * a.heads + h;

  // ---------------------------------------------------------- rows: queries, keys, values, how much is erased, unit keys, decays
  auto load = [&]() {
    bool bad = false;
#pragma unroll 2
    for (int part = 0; part < 4; ++part) {
      const int t = part * 16 + (tid >> 4), c = (tid & 15) * 4;             // sixteen neighbouring lanes a token
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
  float* local = a.local + item * kDcD * kDcD;
  uint32_t* trans = a.trans + item * kTransWords;

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
  if (bad) {
    walk();
    return;
  }

  // ---------------------------------------------------------- decays from the middle: a_s then holds G_t / G_31 for t > 31, its reciprocal up to there
  if (tid < 2 * kDcD) {
    const int c = tid & (kDcD - 1);
    Product p;
    if (tid < kDcD) {
      float w = a_s[31 * kPitchA + c];
      a_s[31 * kPitchA + c] = 1.0f;
#pragma unroll 8
      for (int t = 30; t >= 0; --t) {
        p.times(w);
        w = a_s[t * kPitchA + c];
        a_s[t * kPitchA + c] = p.value();
      }
      p.times(w);
      mid[c] = p.value();                                  // from the stretch's beginning to the middle
    } else {
#pragma unroll 8
      for (int t = 32; t < kChunk; ++t) {
        p.times(a_s[t * kPitchA + c]);
        a_s[t * kPitchA + c] = p.value();
      }
      end[c] = p.value();
    }
  }
  __syncthreads();
  uint32_t largest = 0;                                    // of what is made here to be split
  auto note = [&](float x) { largest = max(largest, magnitude(x)); };
#pragma unroll 4
  for (int e8 = 0; e8 < kChunk * kDcD / kDcThreads; ++e8) {
    const int e = e8 * kDcThreads + tid, t = e >> 6, c = e & 63;
    const float p = a_s[t * kPitchA + c], q = 1.0f / p, f = t > 31 ? p : q, back = t > 31 ? q : p;
    const float before = t == 0 ? 1.0f / mid[c] : (t > 32 ? a_s[(t - 1) * kPitchA + c] : 1.0f / a_s[(t - 1) * kPitchA + c]);
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

  const DcTile w(warp);
  const int lr = lane >> 2, lc = w.c + 2 * (lane & 3);              // a product's numbers: rows + lr and + lr + 8, columns lc + 8 j, + 1
  auto lower = [&](const float* rows, const float* cols, bool strict) {   // a_s = the lower triangle of rows . cols^T
    DcAcc acc = {};
    dc_pairs(acc, rows, cols, w, lane);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      if (w.c > w.row(b)) continue;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = w.row(b) + lr + (i >> 1) * 8, s = lc + j * 8 + (i & 1);
          const float x = (strict ? s < t : s <= t) ? acc[b][j][i] : 0.0f;
          a_s[t * kPitchA + s] = x;
          note(x);
        }
    }
  };
  float* x_s = v_s;                                        // X takes the values' place once they have been used
  DcAcc kv = {}, o = {};
  {
    DcAcc nv = {};
    dc_over_tokens(kv, v_s, k_s, w, lane);                 // [v, k]
    lower(u_s, k_s, true);                                 // N
    __syncthreads();
    dc_times(nv, a_s, v_s, w, lane);
    __syncthreads();
    lower(r_s, k_s, false);                                // A
    __syncthreads();
    dc_times(o, a_s, v_s, w, lane);
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) x_s[(w.row(b) + lr + (i >> 1) * 8) * kDcP + lc + j * 8 + (i & 1)] = nv[b][j][i];
  }
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
    const int c = warp * 16;                               // what these rows take off the ones below, 16 of the 128 columns a warp
    float* tile = (c < kDcD ? x_s : u_s) + (c & (kDcD - 1));
    if (i < 3) {
      FragA fa;
      FragB fb[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) load_b_columns(fb[x], tile + i * 16 * kDcP + x * 8, kDcP, lane);
      for (int j = i + 1; j < 4; ++j) {
        load_a_single(fa, a_s + j * 16 * kPitchA + i * 16, kPitchA, lane);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          float acc[4] = {};
          mma_split(acc, fa, fb[x]);
#pragma unroll
          for (int q = 0; q < 4; ++q) tile[(j * 16 + lr + (q >> 1) * 8) * kDcP + x * 8 + 2 * (lane & 3) + (q & 1)] -= acc[q];
        }
      }
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
    DcAcc bx = {}, bu = {};
    dc_times(bx, a_s, x_s, w, lane);
    dc_times(bu, a_s, u_s, w, lane);
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int t = w.row(b) + lr + half * 8, c = lc + j * 8;
          if (t < n) {
            *reinterpret_cast<float2*>(out + (size_t)t * HD + c) =
                make_float2(o[b][j][2 * half] - bx[b][j][2 * half], o[b][j][2 * half + 1] - bx[b][j][2 * half + 1]);
            *reinterpret_cast<float2*>(reach + (size_t)t * HD + c) =
                make_float2(fmaf(r_s[t * kDcP + c], mid[c], -bu[b][j][2 * half]), fmaf(r_s[t * kDcP + c + 1], mid[c + 1], -bu[b][j][2 * half + 1]));
          }
        }
  }
  {
    DcAcc ex = {}, eu = {};
    dc_over_tokens(ex, x_s, e_s, w, lane);                 // [v, k]
    dc_over_tokens(eu, e_s, u_s, w, lane);                 // [k, k]
    bool lost = false;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int row = w.row(b) + lr + half * 8, c = lc + j * 8;
          *reinterpret_cast<float2*>(local + row * kDcD + c) = make_float2((kv[b][j][2 * half] - ex[b][j][2 * half]) * end[c],
                                                                           (kv[b][j][2 * half + 1] - ex[b][j][2 * half + 1]) * end[c + 1]);
          const float f = end[row], g = f * mid[row];
          eu[b][j][2 * half] = (row == c ? g : 0.0f) - f * eu[b][j][2 * half];
          eu[b][j][2 * half + 1] = (row == c + 1 ? g : 0.0f) - f * eu[b][j][2 * half + 1];
          lost = lost || !splits(eu[b][j][2 * half]) || !splits(eu[b][j][2 * half + 1]);
        }
      Split x[4];
      x[0].set(eu[b][0][0], eu[b][1][0]);
      x[1].set(eu[b][0][2], eu[b][1][2]);
      x[2].set(eu[b][0][1], eu[b][1][1]);
      x[3].set(eu[b][0][3], eu[b][1][3]);
      uint32_t* to = trans + trans_word(w.row(b) >> 4, w.c >> 4, 0, lane);
      *reinterpret_cast<uint4*>(to) = make_uint4(x[0].hi, x[1].hi, x[2].hi, x[3].hi);
      *reinterpret_cast<uint4*>(to + 128) = make_uint4(x[0].mid, x[1].mid, x[2].mid, x[3].mid);
      *reinterpret_cast<uint4*>(to + 256) = make_uint4(x[0].lo, x[1].lo, x[2].lo, x[3].lo);
    }
    lost = __syncthreads_or(lost);
    if (tid == 0) a.bad[item] = lost;
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
  const size_t items = (size_t)chunks * heads, rows = (size_t)num_tokens * heads * kDcD;
  a.local = scratch;
  a.trans = reinterpret_cast<uint32_t*>(a.local + items * kDcD * kDcD);
  a.bad = reinterpret_cast<int*>(a.trans + items * kTransWords);
  a.reach = reinterpret_cast<float*>(a.bad + (items + 3) / 4 * 4);
  a.out = a.reach + rows;
  cudaError_t e = cudaFuncSetAttribute(delta_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DeltaChunkLayout::BYTES);
  if (e != cudaSuccess) return (int)e;
  if (scan_scratch != nullptr) {
    const int rc = launch_delta_scan(proj, ld, w_raw, w0, a_bias, state, slot_stride, cu_seqlens, req_slot, scan_scratch, a.out, num_requests,
                                     num_tokens, heads, dim, min_span - 1, stream);
    if (rc) return rc;
  }
  delta_local_kernel<<<dim3(chunks, heads), kDcThreads, DeltaChunkLayout::BYTES, stream>>>(a);
  IFX_CHECK_LAUNCH();
  delta_carry_kernel<<<dim3(num_requests, heads, kDcD / kCarryV), kCarryThreads, 0, stream>>>(a);
  IFX_CHECK_LAUNCH();
  const int rc = launch_chunk_reach_64(a.reach, a.local, a.out, cu_seqlens, num_requests, min_span, heads, chunks, stream);
  if (rc) return rc;
  return launch_delta_finish(a.out, proj, ld, norm_w, eps, y, num_tokens, heads, dim, out_dtype, stream);
}

}  // extern "C"
