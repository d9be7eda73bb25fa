// Bias add, rotation of queries and keys, and the write of keys and values into
// the paged cache, in one launch.
//
// qkv [T, (nq + 2 nkv) d] holds the stacked projections, either in the run's dtype
// or as float32 partial sums [splits, T, width] of a K-split product, which are
// added here in split order before the bias.  For every token t and
// head: add the bias in float32 (if any), rotate the first `rot` elements of q and
// k heads by angle = position * inv_freq in float32 (precise sincosf), write q to
// q_out [T, nq d], the rotated key and the raw value to the cache page that holds
// the token's position.
//
// Cache layout per layer: [pages, 2 (K, V), nkv, page_size, d].  The page of
// position p of the request in slot s is block_table[s * max_blocks + p / page_size].
#include "common.cuh"

namespace ifx {

template <typename T>
__global__ void rope_append_kernel(const T* __restrict__ qkv, const float* __restrict__ qkv_partial, int num_splits,
                                   size_t split_stride, const float* __restrict__ bias,
                                   const float* __restrict__ inv_freq, int rot, int interleaved,
                                   const int* __restrict__ positions, const int* __restrict__ token_req,
                                   const int* __restrict__ req_slot, const int* __restrict__ block_table,
                                   int max_blocks, int page_size, int num_pages, T* __restrict__ kv_pool,
                                   T* __restrict__ q_out, int nq, int nkv, int d, int write_cache,
                                   int early_dependents) {
  // The attention kernel behind this one is let in early only if the caller says so: a grid of it that fills
  // the SMs would sit on shared memory and fetch keys against the weights of the q/k/v product still running in
  // front (a decode step of the 7B shape at batch 8: 3.07 ms without, 3.24 ms with); a small one gains its
  // prologue (batch 1: 358 against 350 tokens/s).
  if (early_dependents) pdl_launch_dependents();
  // Positions, slots, the block table, the bias and the angles do not come from the kernel in front:
  // they are fetched and the sines computed before it is known to have finished.
  const int t = blockIdx.x;
  const int head = blockIdx.y;                      // [0, nq) q, [nq, nq+nkv) k, then v
  const int width = (nq + 2 * nkv) * d;
  const size_t src_off = (size_t)t * width + (size_t)head * d;
  const T* src = qkv ? qkv + src_off : nullptr;
  const float* psrc = qkv_partial ? qkv_partial + src_off : nullptr;
  auto load2 = [&](int e0, int e1, float& a, float& c) {     // the two elements of a pair, K slices added in order
    if (psrc == nullptr) {
      a = to_f32(src[e0]);
      c = to_f32(src[e1]);
      return;
    }
    a = c = 0.0f;
    for (int s0 = 0; s0 < num_splits; s0 += 8) {                // 16 loads in flight a round
      float va[8], vc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool in = s0 + j < num_splits;
        va[j] = in ? __ldcg(psrc + (size_t)(s0 + j) * split_stride + e0) : 0.0f;
        vc[j] = in ? __ldcg(psrc + (size_t)(s0 + j) * split_stride + e1) : 0.0f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        a += va[j];
        c += vc[j];
      }
    }
  };
  const float* b = bias ? bias + (size_t)head * d : nullptr;
  const int pos = positions[t];

  T* dst = nullptr;
  bool rotate = true;
  if (head < nq) {
    dst = q_out + (size_t)t * nq * d + (size_t)head * d;
  } else if (write_cache) {
    const int is_v = head >= nq + nkv;
    const int g = head - nq - (is_v ? nkv : 0);
    const int slot = req_slot[token_req[t]];
    const int page = block_table[(size_t)slot * max_blocks + pos / page_size];
    if (page >= 0 && page < num_pages)              // never write outside the pool
      dst = kv_pool + ((((size_t)page * 2 + is_v) * nkv + g) * page_size + (pos % page_size)) * d;
    rotate = !is_v;
  }

  const int half_rot = rot / 2;
  struct Pair {
    int e0, e1;
    bool turn;
    float sn, cs, b0, b1;
  };
  auto prepare = [&](int j) -> Pair {
    Pair p;
    p.turn = rotate && j < half_rot;
    if (j < half_rot) {
      p.e0 = interleaved ? 2 * j : j;
      p.e1 = interleaved ? 2 * j + 1 : j + half_rot;
    } else {
      p.e0 = rot + 2 * (j - half_rot);
      p.e1 = p.e0 + 1;
    }
    p.b0 = b ? b[p.e0] : 0.0f;
    p.b1 = b ? b[p.e1] : 0.0f;
    p.sn = 0.0f;
    p.cs = 1.0f;
    if (p.turn) sincosf((float)pos * inv_freq[j], &p.sn, &p.cs);
    return p;
  };
  Pair first = {};
  if ((int)threadIdx.x < d / 2) first = prepare(threadIdx.x);
  pdl_wait();
  if (dst == nullptr) return;
  for (int j = threadIdx.x; j < d / 2; j += blockDim.x) {
    const Pair p = j == (int)threadIdx.x ? first : prepare(j);
    float a, c;
    load2(p.e0, p.e1, a, c);
    a += p.b0;
    c += p.b1;
    if (p.turn) {
      const float ra = a * p.cs - c * p.sn;
      const float rc = a * p.sn + c * p.cs;
      a = ra;
      c = rc;
    }
    if (head >= nq) {                 // the cache only ever holds finite values: a masked key's value gets the
      a = isfinite(a) ? a : 0.0f;     // weight zero, and zero times it must be zero whoever wrote it
      c = isfinite(c) ? c : 0.0f;
    }
    dst[p.e0] = from_f32<T>(a);
    dst[p.e1] = from_f32<T>(c);
  }
}

// The same work for many tokens (prompt portions), TOKENS of them a block.  The cosines and sines of a token's angles are the same for
// all its heads, so they are computed once into shared memory, by as many threads as there are angles; then every thread moves 8 + 8
// elements (a 16-byte chunk and its rotation partner half a head away) of every token per step.  Takes the common case only:
// bfloat16 activations (not partial sums), whole-head split-half rotation, head sizes that are multiples of 16.
// Bound: HBM, and the chains position -> angles and token -> slot -> page, which different warps follow (by one warp after each other they
// took 5 % of a step of prompts' rotations and 20 % where an SM holds one block).  Eight layers of 1,531 tokens, 12 + 4 heads of 128: 52.5 us with a
// token a block, 57.6 with a programmatic launch (EARLY) too, 48.9 with two tokens, 71.5 with four (registers).
template <int TOKENS, bool EARLY>
__global__ void __launch_bounds__(1024)
rope_append_rows_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ bias,
                        const float* __restrict__ inv_freq, const int* __restrict__ positions,
                        const int* __restrict__ token_req, const int* __restrict__ req_slot,
                        const int* __restrict__ block_table, int max_blocks, int page_size, int num_pages,
                        __nv_bfloat16* __restrict__ kv_pool, __nv_bfloat16* __restrict__ q_out, int nq, int nkv, int d,
                        int write_cache, int num_tokens) {
  __shared__ float cs[TOKENS][128], sn[TOKENS][128];    // d / 2 <= 128
  __shared__ long long page_base[TOKENS];               // < 0: no page
  if (EARLY) {
    pdl_launch_dependents();
    pdl_wait();
  }
  const int t0 = blockIdx.x * TOKENS, tokens = min(TOKENS, num_tokens - t0);
  const int half = d / 2;
  const int width = (nq + 2 * nkv) * d;
  const int cph = half / 8;                             // 16-byte chunks per half head
  const int items = (nq + 2 * nkv) * cph;
  const __nv_bfloat16* rows = qkv + (size_t)t0 * width;
  // The block has one thread per item where it can; the item's loads go out before the chains
  // position -> angles and token -> slot -> page are followed.
  int it = threadIdx.x;
  uint4 lo_raw[TOKENS], hi_raw[TOKENS];
  auto fetch = [&](int head, int c) {
#pragma unroll
    for (int k = 0; k < TOKENS; ++k) {
      lo_raw[k] = hi_raw[k] = make_uint4(0u, 0u, 0u, 0u);
      if (k < tokens) {
        lo_raw[k] = *reinterpret_cast<const uint4*>(rows + (size_t)k * width + head * d + c);
        hi_raw[k] = *reinterpret_cast<const uint4*>(rows + (size_t)k * width + head * d + half + c);
      }
    }
  };
  if (it < items) fetch(it / cph, (it % cph) * 8);
  for (int j = threadIdx.x; j < tokens * half; j += blockDim.x) {
    const int k = j / half, a = j - k * half;
    sincosf((float)positions[t0 + k] * inv_freq[a], &sn[k][a], &cs[k][a]);
  }
  const int last = (int)(blockDim.x - 1 - threadIdx.x);    // (not the warps that make angles, if there are others)
  if (last < tokens) {
    long long base = -1;
    if (write_cache) {
      const int t = t0 + last, pos = positions[t], slot = req_slot[token_req[t]];
      const int page = block_table[(size_t)slot * max_blocks + pos / page_size];
      if (page >= 0 && page < num_pages) base = (long long)page * 2 * nkv * page_size * d + (long long)(pos % page_size) * d;
    }
    page_base[last] = base;
  }
  __syncthreads();
  for (; it < items; it += blockDim.x) {
    const int head = it / cph, c = (it % cph) * 8;
    if (it != (int)threadIdx.x) fetch(head, c);          // more items than threads: the later ones load here
    const bool is_q = head < nq, is_v = head >= nq + nkv;
    float blo[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, bhi[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (bias) {                                          // d % 16 == 0: both runs of 8 floats are 32-byte aligned
      const float4* bl = reinterpret_cast<const float4*>(bias + head * d + c);
      const float4* bh = reinterpret_cast<const float4*>(bias + head * d + half + c);
      *reinterpret_cast<float4*>(blo) = bl[0];
      *reinterpret_cast<float4*>(blo + 4) = bl[1];
      *reinterpret_cast<float4*>(bhi) = bh[0];
      *reinterpret_cast<float4*>(bhi + 4) = bh[1];
    }
#pragma unroll
    for (int token = 0; token < TOKENS; ++token) {
      if (token >= tokens) break;
      __nv_bfloat16* dst;
      if (is_q) {
        dst = q_out + (size_t)(t0 + token) * nq * d + (size_t)head * d;
      } else {
        if (page_base[token] < 0) continue;
        const int g = head - nq - (is_v ? nkv : 0);
        dst = kv_pool + page_base[token] + ((size_t)(is_v ? nkv : 0) + g) * page_size * d;
      }
      const __nv_bfloat162* lo2 = reinterpret_cast<const __nv_bfloat162*>(&lo_raw[token]);
      const __nv_bfloat162* hi2 = reinterpret_cast<const __nv_bfloat162*>(&hi_raw[token]);
      uint4 lo_out, hi_out;
      __nv_bfloat162* lo_o = reinterpret_cast<__nv_bfloat162*>(&lo_out);
      __nv_bfloat162* hi_o = reinterpret_cast<__nv_bfloat162*>(&hi_out);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float2 a = __bfloat1622float2(lo2[k]), b = __bfloat1622float2(hi2[k]);
        a.x += blo[2 * k];
        a.y += blo[2 * k + 1];
        b.x += bhi[2 * k];
        b.y += bhi[2 * k + 1];
        if (!is_v) {
          const float2 c2 = *reinterpret_cast<const float2*>(&cs[token][c + 2 * k]), s2 = *reinterpret_cast<const float2*>(&sn[token][c + 2 * k]);
          const float ax = a.x * c2.x - b.x * s2.x, bx = a.x * s2.x + b.x * c2.x;
          const float ay = a.y * c2.y - b.y * s2.y, by = a.y * s2.y + b.y * c2.y;
          a = make_float2(ax, ay);
          b = make_float2(bx, by);
        }
        if (!is_q) {                    // the cache only ever holds finite values
          a.x = isfinite(a.x) ? a.x : 0.0f;
          a.y = isfinite(a.y) ? a.y : 0.0f;
          b.x = isfinite(b.x) ? b.x : 0.0f;
          b.y = isfinite(b.y) ? b.y : 0.0f;
        }
        lo_o[k] = __floats2bfloat162_rn(a.x, a.y);
        hi_o[k] = __floats2bfloat162_rn(b.x, b.y);
      }
      *reinterpret_cast<uint4*>(dst + c) = lo_out;
      *reinterpret_cast<uint4*>(dst + half + c) = hi_out;
    }
  }
}


// The general form for designs whose heads are normed before they are turned, whose values have a size of
// their own, or whose layer stores nothing: one block per (token, head).
//
//   qkv row = [nq heads of d | nkv_src key heads of d | nkv_src value heads of d_v]     (nkv_src may be 0)
//   query and key heads: x / sqrt(mean(x^2) + eps) * w over the head's d elements (w shared by all heads;
//   null: no norm), in float32, before the rotation; then the rotation of the first `rot` elements
//   cache rows have d_row elements (>= d, >= d_v); a key fills the first d, a value the first d_v
template <typename T>
__global__ void norm_rope_append_kernel(const T* __restrict__ qkv, const float* __restrict__ qkv_partial, int num_splits,
                                        size_t split_stride, const float* __restrict__ q_norm_w,
                                        const float* __restrict__ k_norm_w, float norm_eps,
                                        const float* __restrict__ inv_freq, int rot, int interleaved,
                                        const int* __restrict__ positions, const int* __restrict__ token_req,
                                        const int* __restrict__ req_slot, const int* __restrict__ block_table,
                                        int max_blocks, int page_size, int num_pages, T* __restrict__ kv_pool,
                                        T* __restrict__ q_out, int nq, int nkv_src, int nkv_cache, int d, int d_v,
                                        int d_row, int write_cache, float magnitude, float q_temp_coef, int q_temp_every) {
  __shared__ float scratch[32];
  const int t = blockIdx.x;
  const int head = blockIdx.y;                      // [0, nq) q, [nq, nq + nkv_src) k, then v
  const bool is_q = head < nq, is_v = head >= nq + nkv_src;
  const int width = (nq + nkv_src) * d + nkv_src * d_v;
  const int size = is_v ? d_v : d;
  const size_t src_off = (size_t)t * width + (is_v ? (size_t)(nq + nkv_src) * d + (size_t)(head - nq - nkv_src) * d_v
                                                   : (size_t)head * d);
  const int pos = positions[t];
  T* dst = nullptr;
  if (is_q) {
    dst = q_out + ((size_t)t * nq + head) * d;
  } else if (write_cache) {
    const int g = head - nq - (is_v ? nkv_src : 0);
    const int slot = req_slot[token_req[t]];
    const int page = block_table[(size_t)slot * max_blocks + pos / page_size];
    if (page >= 0 && page < num_pages)              // never write outside the pool
      dst = kv_pool + ((((size_t)page * 2 + (is_v ? 1 : 0)) * nkv_cache + g) * page_size + (pos % page_size)) * d_row;
  }
  auto load = [&](int e) -> float {                 // one element, the slices of a K-split product added in order
    if (qkv_partial == nullptr) return to_f32(qkv[src_off + e]);
    float a = 0.0f;
    for (int s0 = 0; s0 < num_splits; ++s0) a += __ldcg(qkv_partial + (size_t)s0 * split_stride + src_off + e);
    return a;
  };
  const float* nw = is_q ? q_norm_w : (is_v ? nullptr : k_norm_w);
  float inv_rms = 1.0f;
  if (nw != nullptr) {                              // every thread of the block takes part in the sum
    float ss = 0.0f;
    for (int e = threadIdx.x; e < size; e += blockDim.x) {
      const float v = load(e);
      ss = fmaf(v, v, ss);
    }
    ss = block_sum(ss, scratch);
    inv_rms = 1.0f / sqrtf(ss / (float)size + norm_eps);
  }
  if (dst == nullptr) return;
  // queries may grow with the position: 1 + coef ln(floor((pos + 1) / every) + 1)
  const float q_mult = (is_q && q_temp_every > 0) ? 1.0f + q_temp_coef * logf((float)((pos + 1) / q_temp_every + 1)) : 1.0f;
  const int half_rot = is_v ? 0 : rot / 2;
  for (int j = threadIdx.x; j < (size + 1) / 2; j += blockDim.x) {
    int e0, e1;
    if (j < half_rot) {
      e0 = interleaved ? 2 * j : j;
      e1 = interleaved ? 2 * j + 1 : j + half_rot;
    } else {
      e0 = 2 * half_rot + 2 * (j - half_rot);
      e1 = e0 + 1;
    }
    float a = load(e0), c = e1 < size ? load(e1) : 0.0f;
    if (nw != nullptr) {
      a = a * inv_rms * nw[e0];
      if (e1 < size) c = c * inv_rms * nw[e1];
    }
    if (j < half_rot) {
      float sn, cs;
      sincosf((float)pos * inv_freq[j], &sn, &cs);
      sn *= magnitude;
      cs *= magnitude;
      const float ra = a * cs - c * sn;
      const float rc = c * cs + a * sn;
      a = ra;
      c = rc;
    }
    a *= q_mult;
    c *= q_mult;
    if (!is_q) {                      // the cache only ever holds finite values
      a = isfinite(a) ? a : 0.0f;
      c = isfinite(c) ? c : 0.0f;
    }
    dst[e0] = from_f32<T>(a);
    if (e1 < size) dst[e1] = from_f32<T>(c);
  }
}

}  // namespace ifx

using namespace ifx;

extern "C" int ifx_rope_append(const void* qkv, const float* qkv_partial, int num_splits, const float* bias, const float* inv_freq, int rot,
                               int interleaved, const int* positions, const int* token_req,
                               const int* req_slot, const int* block_table, int max_blocks, int page_size,
                               int num_pages, void* kv_pool, void* q_out, int num_tokens, int nq, int nkv,
                               int d, int write_cache, int early_dependents, int dtype, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  if (nq <= 0 || nkv <= 0 || d <= 0 || d % 2 || rot < 0 || rot > d || rot % 2) return IFX_E_BADARG;
  if (rot > 0 && inv_freq == nullptr) return IFX_E_BADARG;
  if (write_cache && (page_size <= 0 || max_blocks <= 0 || kv_pool == nullptr)) return IFX_E_BADARG;
  if (nq + 2 * nkv > 65535) return IFX_E_TOOBIG;
  if ((qkv == nullptr) == (qkv_partial == nullptr)) return IFX_E_BADARG;
  if (qkv_partial != nullptr && num_splits <= 0) return IFX_E_BADARG;
  const size_t split_stride = (size_t)num_tokens * (nq + 2 * nkv) * d;
  if (dtype == IFX_DT_BF16 && qkv != nullptr && num_tokens >= 64 && rot == d && !interleaved && d % 16 == 0 &&
      d <= 256 && (reinterpret_cast<uintptr_t>(qkv) % 16 == 0) && (reinterpret_cast<uintptr_t>(q_out) % 16 == 0) &&
      (kv_pool == nullptr || reinterpret_cast<uintptr_t>(kv_pool) % 16 == 0) &&
      (bias == nullptr || reinterpret_cast<uintptr_t>(bias) % 16 == 0)) {
    const int items = (nq + 2 * nkv) * (d / 16);
    const int threads = items >= 1024 ? 1024 : (items + 31) / 32 * 32;
    const dim3 block(threads);
    auto run = [&](auto kern, int tokens) {
      return launch_pdl(kern, dim3((num_tokens + tokens - 1) / tokens), block, 0, stream, 1, (const __nv_bfloat16*)qkv, bias, inv_freq,
                        positions, token_req, req_slot, block_table, max_blocks, page_size, num_pages, (__nv_bfloat16*)kv_pool,
                        (__nv_bfloat16*)q_out, nq, nkv, d, write_cache, num_tokens);
    };
    // More than 512 threads, one block an SM: nothing starts early, and waiting for it costs 4 %.  us, a token a block and two: 64 + 16 heads
    // of 128, 592 tokens 9.0 and 7.1, 2,048 30.1 and 22.4, 8,192 133 and 97; 40 + 80 heads 2,048 43.3 and 34.2.
    if (threads > 512) {
      auto plain = [&](auto kern, int tokens) {
        kern<<<(num_tokens + tokens - 1) / tokens, block, 0, stream>>>(
            (const __nv_bfloat16*)qkv, bias, inv_freq, positions, token_req, req_slot, block_table, max_blocks, page_size, num_pages,
            (__nv_bfloat16*)kv_pool, (__nv_bfloat16*)q_out, nq, nkv, d, write_cache, num_tokens);
        const cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? 0 : (int)e;
      };
      return num_tokens > 148 ? plain(rope_append_rows_kernel<2, false>, 2) : plain(rope_append_rows_kernel<1, false>, 1);
    }
    // Rounds of blocks (an SM holds as many as their 56 or 64 registers a thread let it): one with two tokens a block takes a third longer and
    // more.  us, one and two: 16 heads of 128, 1,000 tokens 3.1 and 3.7, 2,048 4.9 and 4.7, 8,192 14.9 and 14.0; 36 heads 1,000 5.1 and 5.8,
    // 2,048 9.1 and 8.7; 48 of 64, 1,000 4.5 and 4.1; 24 of 256, 592 4.7 and 4.0, 2,048 12.0 and 12.4.
    auto rounds = [&](int registers, int tokens) {
      const int at_once = 148 * tokens * (65536 / (registers * threads));
      return (num_tokens + at_once - 1) / at_once;
    };
    return 4 * rounds(64, 2) < 3 * rounds(56, 1) ? run(rope_append_rows_kernel<2, true>, 2) : run(rope_append_rows_kernel<1, true>, 1);
  }
  dim3 grid(num_tokens, nq + 2 * nkv);
  int threads = d / 2 >= 64 ? 64 : 32;
  if (dtype == IFX_DT_F32)
    return launch_pdl(rope_append_kernel<float>, grid, dim3(threads), 0, stream, 1, (const float*)qkv, qkv_partial,
                      num_splits, split_stride, bias, inv_freq, rot, interleaved, positions, token_req, req_slot,
                      block_table, max_blocks, page_size, num_pages, (float*)kv_pool, (float*)q_out, nq, nkv, d,
                      write_cache, early_dependents);
  if (dtype == IFX_DT_BF16)
    return launch_pdl(rope_append_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream, 1,
                      (const __nv_bfloat16*)qkv, qkv_partial, num_splits, split_stride, bias, inv_freq, rot,
                      interleaved, positions, token_req, req_slot, block_table, max_blocks, page_size, num_pages,
                      (__nv_bfloat16*)kv_pool, (__nv_bfloat16*)q_out, nq, nkv, d, write_cache, early_dependents);
  return IFX_E_DTYPE;
}

// See norm_rope_append_kernel.  nkv_src: key/value heads in the rows of qkv (0: the layer reads another layer's
// cache and projects queries only); nkv_cache: key/value heads of the cache's pages.  magnitude: what cos and sin are
// multiplied by; q_temp_every > 0: queries are multiplied by 1 + q_temp_coef ln(floor((pos + 1) / q_temp_every) + 1).
extern "C" int ifx_norm_rope_append_ex(const void* qkv, const float* qkv_partial, int num_splits, const float* q_norm_w,
                                       const float* k_norm_w, float norm_eps, const float* inv_freq, int rot,
                                       int interleaved, const int* positions, const int* token_req, const int* req_slot,
                                       const int* block_table, int max_blocks, int page_size, int num_pages, void* kv_pool,
                                       void* q_out, int num_tokens, int nq, int nkv_src, int nkv_cache, int d, int d_v,
                                       int d_row, int write_cache, float magnitude, float q_temp_coef, int q_temp_every,
                                       int dtype, cudaStream_t stream) {
  if (q_temp_every < 0) return IFX_E_BADARG;
  if (num_tokens <= 0) return 0;
  if (nq <= 0 || nkv_src < 0 || d <= 0 || d_v <= 0 || rot < 0 || rot > d || rot % 2) return IFX_E_BADARG;
  if (rot > 0 && inv_freq == nullptr) return IFX_E_BADARG;
  if (write_cache && (nkv_src <= 0 || nkv_cache != nkv_src || page_size <= 0 || max_blocks <= 0 || kv_pool == nullptr ||
                      d_row < d || d_row < d_v))
    return IFX_E_BADARG;
  if (nq + 2 * nkv_src > 65535) return IFX_E_TOOBIG;
  if ((qkv == nullptr) == (qkv_partial == nullptr)) return IFX_E_BADARG;
  if (qkv_partial != nullptr && num_splits <= 0) return IFX_E_BADARG;
  const size_t split_stride = (size_t)num_tokens * ((size_t)(nq + nkv_src) * d + (size_t)nkv_src * d_v);
  dim3 grid(num_tokens, nq + 2 * nkv_src);
  const int longest = d > d_v ? d : d_v;
  const int threads = longest / 2 > 64 ? 128 : (longest / 2 > 32 ? 64 : 32);
  if (dtype == IFX_DT_F32)
    norm_rope_append_kernel<float><<<grid, threads, 0, stream>>>(
        (const float*)qkv, qkv_partial, num_splits, split_stride, q_norm_w, k_norm_w, norm_eps, inv_freq, rot,
        interleaved, positions, token_req, req_slot, block_table, max_blocks, page_size, num_pages, (float*)kv_pool,
        (float*)q_out, nq, nkv_src, nkv_cache, d, d_v, d_row, write_cache, magnitude, q_temp_coef, q_temp_every);
  else if (dtype == IFX_DT_BF16)
    norm_rope_append_kernel<__nv_bfloat16><<<grid, threads, 0, stream>>>(
        (const __nv_bfloat16*)qkv, qkv_partial, num_splits, split_stride, q_norm_w, k_norm_w, norm_eps, inv_freq, rot,
        interleaved, positions, token_req, req_slot, block_table, max_blocks, page_size, num_pages,
        (__nv_bfloat16*)kv_pool, (__nv_bfloat16*)q_out, nq, nkv_src, nkv_cache, d, d_v, d_row, write_cache, magnitude,
        q_temp_coef, q_temp_every);
  else
    return IFX_E_DTYPE;
  IFX_CHECK_LAUNCH();
  return 0;
}

extern "C" int ifx_norm_rope_append(const void* qkv, const float* qkv_partial, int num_splits, const float* q_norm_w,
                                    const float* k_norm_w, float norm_eps, const float* inv_freq, int rot,
                                    int interleaved, const int* positions, const int* token_req, const int* req_slot,
                                    const int* block_table, int max_blocks, int page_size, int num_pages, void* kv_pool,
                                    void* q_out, int num_tokens, int nq, int nkv_src, int nkv_cache, int d, int d_v,
                                    int d_row, int write_cache, int dtype, cudaStream_t stream) {
  return ifx_norm_rope_append_ex(qkv, qkv_partial, num_splits, q_norm_w, k_norm_w, norm_eps, inv_freq, rot, interleaved,
                                 positions, token_req, req_slot, block_table, max_blocks, page_size, num_pages, kv_pool,
                                 q_out, num_tokens, nq, nkv_src, nkv_cache, d, d_v, d_row, write_cache, 1.0f, 0.0f, 0, dtype,
                                 stream);
}
