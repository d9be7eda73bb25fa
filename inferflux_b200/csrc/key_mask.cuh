// Which keys a query sees.  Plain arithmetic, for kernels and for the host's compiler alike (tests walk it there).
#pragma once

#ifdef __CUDACC__
#define IFX_BOTH __host__ __device__ __forceinline__
#else
#include <algorithm>
#define IFX_BOTH inline
#endif

namespace ifx {

#ifndef __CUDACC__
using std::max;
using std::min;
#endif

// Which keys a query sees besides "not later than itself": the last `window` of them (> 0), only those of its own
// stretch of `chunk` positions (> 0), or both; the first `keep` keys of a sequence stay visible whatever the window or the
// stretch.  A query's keys are therefore [0, kept(first)) and [first, pos].  `sink`: the softmax's denominator holds one more unit, a key of score 0
// that brings no value; with `sink_values` (one learned number per query head) the unit is exp(that number) instead.
struct KeyMask {
  int window, chunk, sink;
  const float* sink_values;
  int keep;
  // the sink's score in units of log2, for kernels that keep maxima and sums as powers of two
  IFX_BOTH float sink_log2(int head) const {
    return sink_values ? sink_values[head] * 1.4426950408889634f : 0.0f;
  }
  IFX_BOTH int first(int pos) const {          // the first key the query at `pos` sees
    int f = window > 0 ? max(0, pos - window + 1) : 0;
    if (chunk > 0) f = max(f, pos / chunk * chunk);
    return f;
  }
  IFX_BOTH bool any() const { return window > 0 || chunk > 0; }
  IFX_BOTH int kept(int first) const { return min(keep, first); }      // keys in front of `first` that stay
  IFX_BOTH bool sees(int key, int first) const { return key >= first || key < keep; }
};

}  // namespace ifx
