// A mixture of small feed-forward experts: the router's choice and the experts' work for every token.
//
//   moe_route     scores = softmax(z) over all router outputs (float32); the `top` largest of score + correction
//                 are chosen (the earlier index wins a tie); their weights are the scores themselves
//                 (of_chosen: the `top` largest of z + correction are chosen and the weights are the softmax over
//                 the chosen z alone; sigmoid: scores = sigmoid(z), the `top` largest of score + correction are chosen,
//                 and the weights are the chosen scores divided by (their sum + floor))
//   moe_up        act[p] = relu(W_up[e] h[t])^2 for every (token, choice) pair p = t * top + c whose expert e
//                 has weights (experts numbered from `experts` on hand their input on unchanged); or, gated (an
//                 expert's gate rows above its up rows, [experts, 2 ff, width]), with g = min(gate, limit) and
//                 u = clamp(up, -limit, limit): act[p] = g sigmoid(slope g) (u + offset)
//   moe_down      out[t] = sum over the token's choices, in their order, of weight * (W_down[e] act[p]), or
//                 weight * h[t] for an expert without weights
//
// In bfloat16 the work goes one of two ways (the rule and its measurements stand at CudaKernels.moe_kernels): the kernels of this
// file for a little work, sorted rows above.  These sort the (token, choice) pairs by expert first and multiply on the tensor
// cores (gemm_pair_tcgen05.cu):
//
//   moe_sort      every expert's pairs get a stretch of rows, one behind the other, cut into tiles of up to 256 rows of about the
//                 same size; per pair its row (or -1: an expert without weights)
//   moe_gather    rows[row of the pair] = h[token]
//   moe_combine   out[t] = sum over the token's choices, in their order, of weight * y[row of the pair], or
//                 weight * h[t] for an expert without weights
//
// The kernels below the sort are those of the float32 run and of steps with few tokens: a warp makes one output number as a dot
// product (lanes stride the inner size, then a shuffle tree), so every sum has an order that depends on the sizes
// alone.  Expert weights are stacked: up [experts, ff, width], down [experts, width, ff].
#include "common.cuh"
#include "moe_items.cuh"

namespace ifx {

constexpr int kMaxRouterOutputs = 1024;

// One token's choice by a warp: zr its n logits, score_s and choice_s room for n numbers each.
__device__ __forceinline__ void route_token(const float* zr, const float* __restrict__ correction, float* score_s, float* choice_s,
                                            int* __restrict__ ids, float* __restrict__ weights, int n, int top, int of_chosen, float floor,
                                            int lane) {
  const bool sigmoid = of_chosen == 2;
  if (of_chosen == 1) {
    for (int i = lane; i < n; i += 32) {
      score_s[i] = zr[i];
      choice_s[i] = zr[i] + (correction ? correction[i] : 0.0f);
    }
    __syncwarp();
    float m = -INFINITY;                                // the largest chosen logit, known to lane 0
    for (int c = 0; c < top; ++c) {
      float best = -INFINITY;
      int at = 0x7fffffff;
      for (int i = lane; i < n; i += 32) {
        const float v = choice_s[i];
        if (v > best) { best = v; at = i; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
      }
      if (at >= n) at = 0;
      if (lane == 0) {
        ids[c] = at;
        m = fmaxf(m, score_s[at]);
        choice_s[at] = -INFINITY;
      }
      __syncwarp();
    }
    if (lane == 0) {                                     // softmax over the chosen alone, in the order of the choice
      float sum = 0.0f;
      for (int c = 0; c < top; ++c) {
        const float e = expf(score_s[ids[c]] - m);
        weights[c] = e;
        sum += e;
      }
      for (int c = 0; c < top; ++c) weights[c] /= sum;
    }
    return;
  }
  float m = -INFINITY;
  for (int i = lane; i < n; i += 32) m = fmaxf(m, zr[i]);
  m = warp_max(m);
  float sum = 0.0f;
  for (int i = lane; i < n; i += 32) {
    const float e = sigmoid ? 1.0f / (1.0f + expf(-zr[i])) : expf(zr[i] - m);
    score_s[i] = e;
    sum += e;
  }
  sum = sigmoid ? 1.0f : warp_sum(sum);
  for (int i = lane; i < n; i += 32) {
    const float sc = score_s[i] / sum;
    score_s[i] = sc;
    choice_s[i] = sc + (correction ? correction[i] : 0.0f);
  }
  __syncwarp();
  for (int c = 0; c < top; ++c) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int i = lane; i < n; i += 32) {
      const float v = choice_s[i];
      if (v > best) { best = v; at = i; }              // i ascends: the earlier index stays on a tie
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
    if (at >= n) at = 0;                               // only if every score is NaN
    if (lane == 0) {
      ids[c] = at;
      weights[c] = score_s[at];
      choice_s[at] = -INFINITY;
    }
    __syncwarp();
  }
  if (sigmoid && lane == 0) {                            // the chosen scores over their sum, added in the order of the choice
    float total = 0.0f;
    for (int c = 0; c < top; ++c) total += weights[c];
    total += floor;
    for (int c = 0; c < top; ++c) weights[c] /= total;
  }
}

__global__ void moe_route_kernel(const float* __restrict__ z, const float* __restrict__ correction,
                                 int* __restrict__ ids, float* __restrict__ weights, int T, int n, int top, int of_chosen,
                                 float floor) {
  __shared__ float score_s[4][kMaxRouterOutputs];
  __shared__ float choice_s[4][kMaxRouterOutputs];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + warp;
  if (t >= T) return;
  route_token(z + (size_t)t * n, correction, score_s[warp], choice_s[warp], ids + (size_t)t * top, weights + (size_t)t * top, n, top, of_chosen,
              floor, lane);
}

// The same for up to 64 outputs and 32 choices without memory in between: a lane keeps two outputs' scores and one choice.  The largest is
// found by one reduction of ordered bits, and on a tie the earlier index by one vote.
__device__ __forceinline__ void route_token_small(const float* z_s, const float* __restrict__ correction, int* __restrict__ ids,
                                                  float* __restrict__ weights, int n, int top, int of_chosen, float floor, int lane) {
  const unsigned all = 0xffffffffu;
  float score[2], choice[2];
  bool in[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    in[j] = lane + 32 * j < n;
    score[j] = in[j] ? z_s[lane + 32 * j] : -INFINITY;
  }
  if (of_chosen == 2) {
#pragma unroll
    for (int j = 0; j < 2; ++j) score[j] = 1.0f / (1.0f + expf(-score[j]));
  } else if (of_chosen == 0) {
    const float m = warp_max(fmaxf(score[0], score[1]));
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (in[j]) sum += score[j] = expf(score[j] - m);
    sum = warp_sum(sum);
#pragma unroll
    for (int j = 0; j < 2; ++j) score[j] /= sum;
  }
  unsigned key[2];                                         // ordered as the numbers are; 0: not to be chosen (NaN, -inf, chosen before)
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    choice[j] = (in[j] && correction ? score[j] + correction[lane + 32 * j] : score[j]) + 0.0f;       // (one zero)
    const unsigned u = __float_as_uint(choice[j]);
    key[j] = in[j] && choice[j] > -INFINITY ? (u & 0x80000000u ? ~u : u | 0x80000000u) : 0u;
  }
  float mine = -INFINITY;                                  // the lane-th choice's score
  int at_mine = 0;
  for (int c = 0; c < top; ++c) {
    const unsigned best = __reduce_max_sync(all, max(key[0], key[1]));
    const unsigned first = __ballot_sync(all, key[0] == best), second = __ballot_sync(all, key[1] == best);
    const int at = best == 0 ? 0 : first ? __ffs(first) - 1 : 31 + __ffs(second);
    const float s = __shfl_sync(all, at < 32 ? score[0] : score[1], at & 31);
    if (lane == c) mine = s, at_mine = at;
    if (lane == at) key[0] = 0;
    if (lane + 32 == at) key[1] = 0;
  }
  if (of_chosen) {                                         // in the order of the choice
    float m = warp_max(mine), sum = 0.0f;
    if (of_chosen == 1) mine = lane < top ? expf(mine - m) : 0.0f;
    for (int c = 0; c < top; ++c) sum += __shfl_sync(all, mine, c);
    mine /= of_chosen == 2 ? sum + floor : sum;
  }
  if (lane < top) {
    ids[lane] = at_mine;
    weights[lane] = mine;
  }
}

// Router and choice of a bfloat16 step in one launch, up to 64 outputs: 16 tokens a block, whose sixteen warps (eight for more than 32 outputs) share the inner size 32 numbers
// at a time and add up in the order of the warps, so a token's logits depend on nothing else in the step.  A lane reads 16 bytes of a
// row, of which it feeds the first half to one mma.sync of 16 and the second to the next: both operands are permuted alike.
// Bound: latency (the rows' reads, then the choice).  Library product (with its own sum of slices for 18 outputs) and the kernel above -> this,
// us: 24 tokens of 1,536 to 16 outputs 7.2 -> 3.4; 2,048 to 18 12.4 -> 4.1.  More tokens than run at once, and long routers of more than 32
// outputs, are faster by the library (CudaKernels._one_launch_router).
constexpr int kRouterMost = 64, kRouterAhead = 3;
template <int NT>
struct RouterWarps { static constexpr int N = NT <= 4 ? 16 : 8; };      // (shared memory)
template <int NT>
__global__ void __launch_bounds__(RouterWarps<NT>::N * 32) moe_choose_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ w,
                                                                       const float* __restrict__ correction, int* __restrict__ ids,
                                                                       float* __restrict__ weights, int T, int K, int n, int top, int kind,
                                                                       float floor) {
  constexpr int kRouterWarps = RouterWarps<NT>::N;
  __shared__ __align__(16) float part_s[kRouterWarps][16][NT * 8];
  __shared__ float z_s[16][NT * 8], score_s[kRouterWarps][NT * 8], choice_s[kRouterWarps][NT * 8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, t0 = blockIdx.x * 16, units = (K + 31) / 32;
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  uint4 a[kRouterAhead][2], b[kRouterAhead][NT];
  auto column = [&](int u) { return u * 32 + 8 * (lane & 3); };
  auto fetch_w = [&](int u0) {
#pragma unroll
    for (int i = 0; i < kRouterAhead; ++i) {
      const int k = column(u0 + i * kRouterWarps);
#pragma unroll
      for (int j = 0; j < NT; ++j) b[i][j] = k < K && j * 8 + row < n ? __ldg(reinterpret_cast<const uint4*>(w + (size_t)(j * 8 + row) * K + k)) : none;
    }
  };
  fetch_w(warp);                                           // (weights do not come from the kernel in front)
  if (gridDim.x <= 8)                                      // the other rounds' weights on their way into L2: behind a step's experts they
    for (int u = warp + kRouterAhead * kRouterWarps; u < units; u += kRouterWarps) {      // are in DRAM, and few blocks wait for them in turn
      const int k = column(u);
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (k < K && j * 8 + row < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (size_t)(j * 8 + row) * K + k));
    }
  pdl_launch_dependents();
  pdl_wait();
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
  for (int u = warp; u < units; u += kRouterAhead * kRouterWarps) {
#pragma unroll
    for (int i = 0; i < kRouterAhead; ++i) {
      const int k = column(u + i * kRouterWarps);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = t0 + row + 8 * half;
        a[i][half] = k < K && t < T ? *reinterpret_cast<const uint4*>(h + (size_t)t * K + k) : none;
      }
    }
#pragma unroll
    for (int i = 0; i < kRouterAhead; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        auto mma = [&](uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
          asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                       : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                       : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        };
        mma(a[i][0].x, a[i][1].x, a[i][0].y, a[i][1].y, b[i][j].x, b[i][j].y);
        mma(a[i][0].z, a[i][1].z, a[i][0].w, a[i][1].w, b[i][j].z, b[i][j].w);
      }
    if (u + kRouterAhead * kRouterWarps < units) fetch_w(u + kRouterAhead * kRouterWarps);
  }
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    float* to = &part_s[warp][row][j * 8 + 2 * (lane & 3)];
    *reinterpret_cast<float2*>(to) = make_float2(acc[j][0], acc[j][1]);
    *reinterpret_cast<float2*>(to + 8 * NT * 8) = make_float2(acc[j][2], acc[j][3]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * NT * 8; i += kRouterWarps * 32) {
    float z = (&part_s[0][0][0])[i];
#pragma unroll
    for (int v = 1; v < kRouterWarps; ++v) z += (&part_s[v][0][0])[i];
    (&z_s[0][0])[i] = z;
  }
  __syncthreads();
  for (int i = warp; i < 16 && t0 + i < T; i += kRouterWarps) {
    int* to = ids + (size_t)(t0 + i) * top;
    float* wt = weights + (size_t)(t0 + i) * top;
    if (top <= 32) {
      route_token_small(z_s[i], correction, to, wt, n, top, kind, floor, lane);
    } else {
      route_token(z_s[i], correction, score_s[warp], choice_s[warp], to, wt, n, top, kind, floor, lane);
      __syncwarp();
    }
  }
}

template <typename T>
__device__ __forceinline__ float dot_lanes(const T* __restrict__ w, const float* __restrict__ a, int n, int lane) {
  float s = 0.0f;
  for (int i = lane; i < n; i += 32) s = fmaf(to_f32(w[i]), a[i], s);
  return warp_sum(s);
}

// bfloat16 weights in 16-byte pieces, four of them in flight per lane, when the row allows it.
template <>
__device__ __forceinline__ float dot_lanes<__nv_bfloat16>(const __nv_bfloat16* __restrict__ w, const float* __restrict__ a,
                                                          int n, int lane) {
  float s = 0.0f;
  if ((n & 7) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
    const uint4* w8 = reinterpret_cast<const uint4*>(w);
    const int chunks = n >> 3;
    auto use = [&](uint4 raw, int chunk) {
      const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
      const float4 a0 = *reinterpret_cast<const float4*>(a + 8 * chunk), a1 = *reinterpret_cast<const float4*>(a + 8 * chunk + 4);
      const float2 f0 = __bfloat1622float2(p2[0]), f1 = __bfloat1622float2(p2[1]);
      const float2 f2 = __bfloat1622float2(p2[2]), f3 = __bfloat1622float2(p2[3]);
      s = fmaf(f0.x, a0.x, s); s = fmaf(f0.y, a0.y, s); s = fmaf(f1.x, a0.z, s); s = fmaf(f1.y, a0.w, s);
      s = fmaf(f2.x, a1.x, s); s = fmaf(f2.y, a1.y, s); s = fmaf(f3.x, a1.z, s); s = fmaf(f3.y, a1.w, s);
    };
    int i = lane;
    for (; i + 96 < chunks; i += 128) {
      const uint4 r0 = __ldg(w8 + i), r1 = __ldg(w8 + i + 32), r2 = __ldg(w8 + i + 64), r3 = __ldg(w8 + i + 96);
      use(r0, i); use(r1, i + 32); use(r2, i + 64); use(r3, i + 96);
    }
    for (; i < chunks; i += 32) use(__ldg(w8 + i), i);
  } else {
    for (int i = lane; i < n; i += 32) s = fmaf(__bfloat162float(w[i]), a[i], s);
  }
  return warp_sum(s);
}

// NR rows of bfloat16 weights against the same staged vector, their 16-byte loads in flight together (a row alone
// leaves a lane with too few bytes under way to keep the memory busy).  Each row's sum is added in the order dot_lanes uses.
template <int NR>
__device__ __forceinline__ void dot_lanes_rows(const __nv_bfloat16* const (&w)[NR], const float* __restrict__ a, int n,
                                               int lane, float (&out)[NR]) {
  float s[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) s[r] = 0.0f;
  bool wide = (n & 7) == 0;
#pragma unroll
  for (int r = 0; r < NR; ++r) wide = wide && (reinterpret_cast<uintptr_t>(w[r]) & 15) == 0;
  if (wide) {
    const int chunks = n >> 3;
    auto use = [&](uint4 raw, int chunk, float& acc) {
      const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
      const float4 a0 = *reinterpret_cast<const float4*>(a + 8 * chunk), a1 = *reinterpret_cast<const float4*>(a + 8 * chunk + 4);
      const float2 f0 = __bfloat1622float2(p2[0]), f1 = __bfloat1622float2(p2[1]);
      const float2 f2 = __bfloat1622float2(p2[2]), f3 = __bfloat1622float2(p2[3]);
      acc = fmaf(f0.x, a0.x, acc); acc = fmaf(f0.y, a0.y, acc); acc = fmaf(f1.x, a0.z, acc); acc = fmaf(f1.y, a0.w, acc);
      acc = fmaf(f2.x, a1.x, acc); acc = fmaf(f2.y, a1.y, acc); acc = fmaf(f3.x, a1.z, acc); acc = fmaf(f3.y, a1.w, acc);
    };
    int i = lane;
    for (; i + 32 < chunks; i += 64) {
      uint4 lo[NR], hi[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        lo[r] = __ldg(reinterpret_cast<const uint4*>(w[r]) + i);
        hi[r] = __ldg(reinterpret_cast<const uint4*>(w[r]) + i + 32);
      }
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        use(lo[r], i, s[r]);
        use(hi[r], i + 32, s[r]);
      }
    }
    for (; i < chunks; i += 32) {
      uint4 lo[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) lo[r] = __ldg(reinterpret_cast<const uint4*>(w[r]) + i);
#pragma unroll
      for (int r = 0; r < NR; ++r) use(lo[r], i, s[r]);
    }
  } else {
    for (int i = lane; i < n; i += 32) {
#pragma unroll
      for (int r = 0; r < NR; ++r) s[r] = fmaf(__bfloat162float(w[r][i]), a[i], s[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r) out[r] = warp_sum(s[r]);
}

template <int NR>
__device__ __forceinline__ void dot_lanes_rows(const float* const (&w)[NR], const float* __restrict__ a, int n, int lane,
                                               float (&out)[NR]) {
#pragma unroll
  for (int r = 0; r < NR; ++r) out[r] = dot_lanes<float>(w[r], a, n, lane);
}

constexpr int kMoeWarps = 8;

template <typename T, bool GLU>
__global__ void moe_up_kernel(const T* __restrict__ h, const T* __restrict__ w_up, const int* __restrict__ ids,
                              T* __restrict__ act, int top, int experts, int width, int ff, int rows_per_block,
                              float limit, float slope, float offset) {
  extern __shared__ __align__(16) float h_s[];
  const int p = blockIdx.x;
  const int e = ids[p];
  if (e >= experts || e < 0) return;
  const int t = p / top;
  for (int i = threadIdx.x; i < width; i += blockDim.x) h_s[i] = to_f32(h[(size_t)t * width + i]);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int f0 = blockIdx.y * rows_per_block;
  const T* w = w_up + (size_t)e * (GLU ? 2 : 1) * ff * width;
  const int last = min(ff, f0 + rows_per_block) - 1;
  for (int f = f0 + warp; f <= last; f += 4 * kMoeWarps) {           // four rows of a warp at a time
    const T* rows[4];
    float z[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) rows[r] = w + (size_t)min(f + r * kMoeWarps, last) * width;
    dot_lanes_rows<4>(rows, h_s, width, lane, z);
    if (GLU) {
      float up[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) rows[r] += (size_t)ff * width;     // the up rows lie ff rows below the gate rows
      dot_lanes_rows<4>(rows, h_s, width, lane, up);
      if (lane == 0) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float g = fminf(z[r], limit), u = fminf(fmaxf(up[r], -limit), limit);
          if (f + r * kMoeWarps <= last)
            act[(size_t)p * ff + f + r * kMoeWarps] = from_f32<T>(g / (1.0f + expf(-slope * g)) * (u + offset));
        }
      }
      continue;
    }
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float zf = fmaxf(z[r], 0.0f);
        if (f + r * kMoeWarps <= last) act[(size_t)p * ff + f + r * kMoeWarps] = from_f32<T>(zf * zf);
      }
    }
  }
}

template <typename T, typename TO>
__global__ void moe_down_kernel(const T* __restrict__ h, const T* __restrict__ act, const T* __restrict__ w_down,
                                const int* __restrict__ ids, const float* __restrict__ weights, TO* __restrict__ out,
                                int top, int experts, int width, int ff, int rows_per_block) {
  extern __shared__ __align__(16) float a_s[];
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.y * rows_per_block, c1 = min(width, c0 + rows_per_block);
  float acc[8];                                         // rows c0 + warp + 8 r of this warp
#pragma unroll
  for (int r = 0; r < 8; ++r) acc[r] = 0.0f;
  for (int c = 0; c < top; ++c) {
    const int p = t * top + c;
    const int e = ids[p];
    const float g = weights[p];
    if (e >= experts || e < 0) {                        // the input itself
      if (lane == 0) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int row = c0 + warp + kMoeWarps * r;
          if (row < c1) acc[r] = fmaf(g, to_f32(h[(size_t)t * width + row]), acc[r]);
        }
      }
      continue;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ff; i += blockDim.x) a_s[i] = to_f32(act[(size_t)p * ff + i]);
    __syncthreads();
    const T* w = w_down + (size_t)e * width * ff;
#pragma unroll
    for (int r0 = 0; r0 < 8; r0 += 4) {
      if (c0 + warp + kMoeWarps * r0 >= c1) break;
      const T* rows[4];
      float d[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) rows[r] = w + (size_t)min(c0 + warp + kMoeWarps * (r0 + r), c1 - 1) * ff;
      dot_lanes_rows<4>(rows, a_s, ff, lane, d);
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (c0 + warp + kMoeWarps * (r0 + r) < c1) acc[r0 + r] = fmaf(g, d[r], acc[r0 + r]);
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int row = c0 + warp + kMoeWarps * r;
      if (row < c1) out[(size_t)t * width + row] = from_f32<TO>(acc[r]);
    }
  }
}

// One block.  Pairs of one expert inside a warp draw their places with one addition (an addition a pair: 8,192 pairs of 16 experts
// 10.7 us, so 5.0); experts' stretches are found by a scan over all of them (one thread walking 1,024 experts: 20 us more).
__global__ void __launch_bounds__(1024) moe_sort_kernel(const int* __restrict__ ids, int pairs, int experts, PairItem* __restrict__ items,
                                                        int* __restrict__ pair_row) {
  static_assert(kMaxRouterOutputs == 1024, "a thread an expert");
  __shared__ int count_s[kMaxRouterOutputs], row_s[kMaxRouterOutputs], warp_rows[32], warp_items[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  count_s[threadIdx.x] = 0;
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait();
  for (int p0 = 0; p0 < pairs; p0 += 1024) {
    const int p = p0 + threadIdx.x;
    int e = p < pairs ? ids[p] : -1;
    if (e < 0 || e >= experts) e = -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    int base = 0;
    if (e >= 0 && lane == __ffs(same) - 1) base = atomicAdd(&count_s[e], __popc(same));
    base = __shfl_sync(0xffffffffu, base, __ffs(same) - 1);
    // which row inside the stretch does not change a row's result
    if (p < pairs) pair_row[p] = e >= 0 ? base + __popc(same & ((1u << lane) - 1)) : -1;
  }
  __syncthreads();
  const int count = count_s[threadIdx.x], tiles = (count + kItemTokens - 1) / kItemTokens;
  int rows_to = count, items_to = tiles;                     // sums up to and with this expert
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int r = __shfl_up_sync(0xffffffffu, rows_to, o), i = __shfl_up_sync(0xffffffffu, items_to, o);
    if (lane >= o) rows_to += r, items_to += i;
  }
  if (lane == 31) warp_rows[warp] = rows_to, warp_items[warp] = items_to;
  __syncthreads();
  int rows_before = 0, items_before = 0;
  for (int w = 0; w < warp; ++w) rows_before += warp_rows[w], items_before += warp_items[w];
  const int first = rows_before + rows_to - count;
  row_s[threadIdx.x] = first;
  int at = 1 + items_before + items_to - tiles, begin = 0;
  for (int i = 0; i < tiles; ++i) {                          // the tiles' sizes differ by one at most
    const int n = (count - begin + tiles - i - 1) / (tiles - i);
    items[at + i] = PairItem{(int)threadIdx.x, first + begin, n, (n + 31) / 32 * 32};
    begin += n;
  }
  if (threadIdx.x == 1023) items[0] = PairItem{items_before + items_to, 0, 0, 0};
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += 1024) {
    const int place = pair_row[p];
    if (place >= 0) pair_row[p] = row_s[ids[p]] + place;
  }
}

// A block a token: its row is read once.
__global__ void moe_gather_kernel(const __nv_bfloat16* __restrict__ h, const int* __restrict__ pair_row,
                                  __nv_bfloat16* __restrict__ rows, int top, int width8) {
  pdl_launch_dependents();
  pdl_wait();
  const uint4* src = reinterpret_cast<const uint4*>(h) + (size_t)blockIdx.x * width8;
  const int* row = pair_row + (size_t)blockIdx.x * top;
  for (int i = threadIdx.x; i < width8; i += blockDim.x) {
    const uint4 v = src[i];
    for (int k = 0; k < top; ++k)
      if (row[k] >= 0) reinterpret_cast<uint4*>(rows)[(size_t)row[k] * width8 + i] = v;
  }
}

constexpr int kMoeSlices = 3;          // of a few tokens' second product at most
// Eight columns a thread: two loads of 16 bytes a choice and slice, all choices' in flight.  SLICED: y is [slices, rows, width]
// (24 tokens, four choices of three slices 7.0 us with a loop of loads and additions, so 5.2).
template <typename TO, bool SLICED>
__global__ void moe_combine_kernel(const __nv_bfloat16* __restrict__ h, const float* __restrict__ y,
                                   const float* __restrict__ weights, const int* __restrict__ pair_row, TO* __restrict__ out,
                                   int top, int width, int slices) {
  pdl_wait();
  const int t = blockIdx.x;
  const size_t slice = (size_t)gridDim.x * top * width;
  for (int c = threadIdx.x * 8; c < width; c += blockDim.x * 8) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
#pragma unroll 4
    for (int k = 0; k < top; ++k) {
      const int p = t * top + k, row = pair_row[p];
      const float w = weights[p];
      if (row >= 0) {                                        // a product, then a sum, each rounded: the same sums however K is cut
        constexpr int MOST = SLICED ? kMoeSlices : 1;
        const float* src = y + (size_t)row * width + c;
        float v[MOST][8];
#pragma unroll
        for (int s = 0; s < MOST; ++s) {                     // (the last slice again for one that is not there)
          const float4* at = reinterpret_cast<const float4*>(src + (SLICED ? min(s, slices - 1) * slice : 0));
          reinterpret_cast<float4*>(v[s])[0] = at[0];
          reinterpret_cast<float4*>(v[s])[1] = at[1];
        }
#pragma unroll
        for (int s = 0; s < MOST; ++s)
          if (!SLICED || s < slices) {
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(acc[i], __fmul_rn(v[s][i], w));
          }
      } else {
        const uint4 raw = *reinterpret_cast<const uint4*>(h + (size_t)t * width + c);
        const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, to_f32(b[i]), acc[i]);
      }
    }
    TO* dst = out + (size_t)t * width + c;
    if constexpr (sizeof(TO) == 4) {
      reinterpret_cast<float4*>(dst)[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      reinterpret_cast<float4*>(dst)[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
      __nv_bfloat162 b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) b[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(b);
    }
  }
}

int gemm_pair(int mode, const void* tokens, const void* W, void* out, int rows, int N, int K, int stack, const PairItem* items,
              int most_items, int slice_kblocks, float limit, float slope, float offset, int* error_flag, cudaStream_t stream);

static long long moe_aligned(long long bytes) { return (bytes + 255) / 256 * 256; }
static int moe_most_items(int pairs, int experts) { return pairs / kItemTokens + (experts < pairs ? experts : pairs); }

// Slices of K of a few tokens' second product: three, or one of a short K.  None is empty.
static int moe_slice_kblocks(int ff) {
  const int kblocks = (ff + 63) / 64, want = kblocks < 12 ? 1 : kMoeSlices;
  return (kblocks + want - 1) / want;
}
static int moe_slices(int ff, int few) { return few ? ((ff + 63) / 64 + moe_slice_kblocks(ff) - 1) / moe_slice_kblocks(ff) : 1; }

}  // namespace ifx

using namespace ifx;

extern "C" {

// kind: 0 softmax over all, 1 softmax over the chosen, 2 sigmoid scores over the chosen scores' sum + floor.
int ifx_moe_route_kind(const float* z, const float* correction, int* ids, float* weights, int T, int n, int top,
                       int kind, float floor, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (n <= 0 || top <= 0 || top > n || kind < 0 || kind > 2) return IFX_E_BADARG;
  if (n > kMaxRouterOutputs) return IFX_E_TOOBIG;
  moe_route_kernel<<<(T + 3) / 4, 128, 0, stream>>>(z, correction, ids, weights, T, n, top, kind, floor);
  IFX_CHECK_LAUNCH();
  return 0;
}

// The same with the router in front of it: z = h [T, K] . w [n, K]^T, both bfloat16 on 16-byte boundaries, K a multiple of 8, n up to 64.
int ifx_moe_choose(const void* h, const void* w, const float* correction, int* ids, float* weights, int T, int K, int n, int top, int kind,
                   float floor, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (K <= 0 || K % 8 || n <= 0 || top <= 0 || top > n || kind < 0 || kind > 2) return IFX_E_BADARG;
  if (n > kRouterMost) return IFX_E_TOOBIG;
  if (((uintptr_t)h | (uintptr_t)w) % 16) return IFX_E_ALIGN;
  auto run = [&](auto kern, int warps = 16) {
    return launch_pdl(kern, dim3((T + 15) / 16), dim3(warps * 32), 0, stream, 1, (const __nv_bfloat16*)h, (const __nv_bfloat16*)w, correction,
                      ids, weights, T, K, n, top, kind, floor);
  };
  if (n <= 8) return run(moe_choose_kernel<1>);
  if (n <= 16) return run(moe_choose_kernel<2>);
  if (n <= 24) return run(moe_choose_kernel<3>);
  if (n <= 32) return run(moe_choose_kernel<4>);
  return run(moe_choose_kernel<8>, RouterWarps<8>::N);
}

int ifx_moe_route_ex(const float* z, const float* correction, int* ids, float* weights, int T, int n, int top,
                     int of_chosen, cudaStream_t stream) {
  return ifx_moe_route_kind(z, correction, ids, weights, T, n, top, of_chosen ? 1 : 0, 0.0f, stream);
}

int ifx_moe_route(const float* z, const float* correction, int* ids, float* weights, int T, int n, int top,
                  cudaStream_t stream) {
  return ifx_moe_route_ex(z, correction, ids, weights, T, n, top, 0, stream);
}

// h [T, width], act [T * top, ff] in `dtype`; out [T, width] in out_dtype.
int ifx_moe_experts_ex(const void* h, const void* w_up, const void* w_down, const int* ids, const float* weights,
                       void* act, void* out, int T, int top, int experts, int width, int ff, int dtype, int out_dtype,
                       int glu, float limit, float slope, cudaStream_t stream);
int ifx_moe_experts_glu(const void* h, const void* w_up, const void* w_down, const int* ids, const float* weights,
                        void* act, void* out, int T, int top, int experts, int width, int ff, int dtype, int out_dtype,
                        int glu, float limit, float slope, float offset, cudaStream_t stream);

int ifx_moe_experts(const void* h, const void* w_up, const void* w_down, const int* ids, const float* weights,
                    void* act, void* out, int T, int top, int experts, int width, int ff, int dtype, int out_dtype,
                    cudaStream_t stream) {
  return ifx_moe_experts_ex(h, w_up, w_down, ids, weights, act, out, T, top, experts, width, ff, dtype, out_dtype, 0, 0.0f,
                            0.0f, stream);
}

int ifx_moe_experts_ex(const void* h, const void* w_up, const void* w_down, const int* ids, const float* weights,
                       void* act, void* out, int T, int top, int experts, int width, int ff, int dtype, int out_dtype,
                       int glu, float limit, float slope, cudaStream_t stream) {
  return ifx_moe_experts_glu(h, w_up, w_down, ids, weights, act, out, T, top, experts, width, ff, dtype, out_dtype, glu, limit,
                             slope, 1.0f, stream);
}

// glu: w_up is [experts, 2 ff, width], an expert's gate rows above its up rows, and the activation is the gated one,
// g sigmoid(slope g) (u + offset) with g cut at limit from above and u on both sides (limit +inf: nothing is cut).
int ifx_moe_experts_glu(const void* h, const void* w_up, const void* w_down, const int* ids, const float* weights,
                        void* act, void* out, int T, int top, int experts, int width, int ff, int dtype, int out_dtype,
                        int glu, float limit, float slope, float offset, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (top <= 0 || experts < 0 || width <= 0 || ff <= 0) return IFX_E_BADARG;
  if ((size_t)width * 4 > 160 * 1024 || (size_t)ff * 4 > 160 * 1024) return IFX_E_TOOBIG;
  const int up_rows = 32, down_rows = T <= 64 ? 32 : 64;  // few tokens: more blocks, so that more bytes are in flight
  dim3 grid_up(T * top, (ff + up_rows - 1) / up_rows), grid_down(T, (width + down_rows - 1) / down_rows);
  const size_t smem_up = (size_t)width * 4, smem_down = (size_t)ff * 4;
#define IFX_MOE(TT, TO)                                                                                           \
  do {                                                                                                            \
    if (experts > 0) {                                                                                            \
      auto up = glu ? moe_up_kernel<TT, true> : moe_up_kernel<TT, false>;                                         \
      if (smem_up > 48 * 1024) cudaFuncSetAttribute(up, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_up); \
      up<<<grid_up, kMoeWarps * 32, smem_up, stream>>>((const TT*)h, (const TT*)w_up, ids, (TT*)act, top, experts, \
                                                       width, ff, up_rows, limit, slope, offset);                         \
    }                                                                                                             \
    auto down = moe_down_kernel<TT, TO>;                                                                          \
    if (smem_down > 48 * 1024)                                                                                    \
      cudaFuncSetAttribute(down, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_down);                    \
    down<<<grid_down, kMoeWarps * 32, smem_down, stream>>>((const TT*)h, (const TT*)act, (const TT*)w_down, ids,  \
                                                           weights, (TO*)out, top, experts, width, ff, down_rows); \
  } while (0)
  if (dtype == IFX_DT_F32 && out_dtype == IFX_DT_F32) IFX_MOE(float, float);
  else if (dtype == IFX_DT_BF16 && out_dtype == IFX_DT_BF16) IFX_MOE(__nv_bfloat16, __nv_bfloat16);
  else if (dtype == IFX_DT_BF16 && out_dtype == IFX_DT_F32) IFX_MOE(__nv_bfloat16, float);
  else return IFX_E_DTYPE;
#undef IFX_MOE
  IFX_CHECK_LAUNCH();
  return 0;
}

// Bytes of scratch of ifx_moe_sorted: the list of tiles, the pairs' rows, gathered rows, activations, the experts' outputs.
long long ifx_moe_sorted_scratch(int T, int top, int experts, int width, int ff, int few) {
  const long long pairs = (long long)T * top;
  return moe_aligned((1 + moe_most_items((int)pairs, experts)) * (long long)sizeof(PairItem)) + moe_aligned(pairs * 4) +
         moe_aligned(pairs * width * 2) + moe_aligned(pairs * ff * 2) + pairs * width * 4 * moe_slices(ff, few);
}

// The experts of a bfloat16 step over sorted rows.  h [T, width]; w_up [experts, ff, width] (glu: [experts, 2 ff, width], gate rows
// above up rows); w_down [experts, width, ff]; ids, weights [T, top]; out [T, width] in out_dtype.  width and ff multiples of 8;
// matrices, h, out and scratch on 16-byte boundaries.  few: a step of few tokens, whose second product's K is cut into slices that
// are added in float32, and whose gates' exponentials and divisions are not the fast ones.
int ifx_moe_sorted(const void* h, const void* w_up, const void* w_down, const int* ids, const float* weights, void* out, int T, int top,
                   int experts, int width, int ff, int out_dtype, int glu, int few, float limit, float slope, float offset,
                   void* scratch, long long scratch_bytes, int* error_flag, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (top <= 0 || experts <= 0 || experts > kMaxRouterOutputs || width <= 0 || ff <= 0 || width % 8 || ff % 8 || error_flag == nullptr)
    return IFX_E_BADARG;
  if (out_dtype != IFX_DT_F32 && out_dtype != IFX_DT_BF16) return IFX_E_DTYPE;
  if (((uintptr_t)h | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)out | (uintptr_t)scratch) % 16) return IFX_E_ALIGN;
  if ((long long)T * top > 0x7fffffffll || scratch_bytes < ifx_moe_sorted_scratch(T, top, experts, width, ff, few)) return IFX_E_TOOBIG;
  const int pairs = T * top, most = moe_most_items(pairs, experts);
  unsigned char* at = reinterpret_cast<unsigned char*>(scratch);
  auto take = [&](long long bytes) {
    unsigned char* p = at;
    at += moe_aligned(bytes);
    return p;
  };
  PairItem* items = reinterpret_cast<PairItem*>(take((1 + most) * (long long)sizeof(PairItem)));
  int* pair_row = reinterpret_cast<int*>(take(pairs * 4ll));
  __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(take((long long)pairs * width * 2));
  __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(take((long long)pairs * ff * 2));
  float* y = reinterpret_cast<float*>(at);
  int rc = launch_pdl(moe_sort_kernel, dim3(1), dim3(1024), 0, stream, 1, ids, pairs, experts, items, pair_row);
  if (rc) return rc;
  rc = launch_pdl(moe_gather_kernel, dim3(T), dim3(192), 0, stream, 1, (const __nv_bfloat16*)h, pair_row, rows, top, width / 8);
  if (rc) return rc;
  rc = gemm_pair(!glu ? 0 : few ? 4 : 2, rows, w_up, act, pairs, ff, width, experts, items, most, 0, limit, slope, offset, error_flag, stream);
  if (rc) return rc;
  const int slices = moe_slices(ff, few), per = slices > 1 ? moe_slice_kblocks(ff) : 0;
  rc = gemm_pair(1, act, w_down, y, pairs, width, ff, experts, items, most, per, 0.0f, 0.0f, 0.0f, error_flag, stream);
  if (rc) return rc;
  const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(h);
#define IFX_COMBINE(TO, SLICED)                                                                                                      \
  launch_pdl(moe_combine_kernel<TO, SLICED>, dim3(T), dim3(192), 0, stream, 1, hb, y, weights, pair_row, (TO*)out, top, width, slices)
  if (out_dtype == IFX_DT_BF16) return slices > 1 ? IFX_COMBINE(__nv_bfloat16, true) : IFX_COMBINE(__nv_bfloat16, false);
  return slices > 1 ? IFX_COMBINE(float, true) : IFX_COMBINE(float, false);
#undef IFX_COMBINE
}

}  // extern "C"
