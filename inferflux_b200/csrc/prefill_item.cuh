// What a block of prompt attention's grid (attention_tcgen05.cu) has to do: its query tiles and the key tiles it walks.  Plain
// arithmetic, for the kernel and for the host's compiler alike (tests walk it there).
#pragma once

#include "key_mask.cuh"

#ifndef __CUDACC__
struct float2;
#endif

namespace ifx {

constexpr int kBM = 128;      // queries per tile
constexpr int kBN = 128;      // keys per tile

// What is left over when whole rounds of blocks, one an SM, have been taken off a grid runs as `parts` blocks each, every one over a
// part of the keys, and leaves an unnormalised sum, its reference and its denominator for prefill_merge_kernel.  A plain grid has
// full = its blocks.  (28 heads x 11 items on 148 SMs are two rounds and 12 blocks, which alone took a third round.)
struct PrefillParts {
  int full, parts;
  int halves;                // 1: the grid has a block for each of an item's query tiles (parts is 1)
  float* o;                  // [left over x parts][256][D]
  float2* ml;                // [left over x parts][256]: reference in units of log2, sum
};

// What a block of the grid has to do.  KEPT: the mask has kept first keys (without them the walk over the key tiles is a plain range).
template <bool KEPT>
struct PrefillItem {
  int r, row0, rows, pos0, h, slot;        // request, rows of the step, position of the first; slot < 0: a block with all of its keys
  int rows_1;                              // rows of query tile 1
  int tb_0, te_0, tb_1, te_1, te;          // key tiles [tb_q, te_q) of query tile q (rows q * 128 ...); tile 1 may be absent
  int keep, keep_tiles, nk, tb;

  IFX_BOTH PrefillItem(int block, const int* tiles, int num_tiles, int nq, const KeyMask& window, const PrefillParts& split) {
    // the last items of a prompt see the most keys: they go first; the heads of an item run side by side
    int part = 0;
    slot = block - split.full;
    if (slot >= 0) {
      block = split.full + slot / split.parts;
      part = slot % split.parts;
    }
    int half = 0;                                          // (an item's second tile sees more keys: it goes first)
    if (split.halves) {
      half = 1 - block / nq % 2;
      block = block / (2 * nq) * nq + block % nq;
    }
    const int* tile = tiles + (size_t)(num_tiles - 1 - block / nq) * 4;
    r = tile[0], row0 = tile[1] + half * kBM, rows = tile[2] - half * kBM, pos0 = tile[3] + half * kBM;
    if (split.halves) rows = min(max(rows, 0), kBM);
    h = block % nq;
    rows_1 = max(rows - kBM, 0);
    tb_0 = window.first(pos0) / kBN;
    te_0 = (pos0 + min(rows, kBM) + kBN - 1) / kBN;
    tb_1 = window.first(pos0 + kBM) / kBN;
    te_1 = rows_1 > 0 ? (pos0 + rows + kBN - 1) / kBN : tb_1;
    if (!KEPT && slot >= 0) {                              // this block's part of the key tiles (tile 0 begins first)
      const int last = max(te_0, te_1), per = (last - tb_0 + split.parts - 1) / split.parts;
      const int lo = min(last, tb_0 + part * per), hi = min(last, lo + per);
      tb_0 = lo;
      te_0 = max(lo, min(te_0, hi));
      tb_1 = max(lo, min(tb_1, hi));
      te_1 = max(tb_1, min(te_1, hi));
    }
    if (rows == 0) te_0 = tb_1 = te_1 = tb_0;              // a second query tile that is not there: no key tile is walked for it
    te = max(te_0, te_1);
    // Key tiles are visited in order: with kept keys first [0, nk), then [tb_0, te); query tile q uses those that hold kept keys
    // and those of its own window.
    keep = KEPT ? window.keep : 0, keep_tiles = (keep + kBN - 1) / kBN, nk = min(keep_tiles, tb_0);
    tb = KEPT && nk > 0 ? 0 : tb_0;
  }
  IFX_BOTH int next_tile(int kt) const { return KEPT && kt + 1 == nk ? tb_0 : kt + 1; }
  IFX_BOTH int visited(int kt) const { return KEPT && kt < nk ? kt : kt - tb_0 + nk; }   // tiles that come before kt
  IFX_BOTH int visits() const { return te - tb_0 + nk; }
  IFX_BOTH bool active(int q, int kt) const {
    if (KEPT && kt < keep_tiles && kt < te_0 && (q == 0 || rows_1 > 0)) return true;      // (kept keys lie in front of te_0)
    return q == 0 ? (kt >= tb_0 && kt < te_0) : (kt >= tb_1 && kt < te_1);
  }
  IFX_BOTH bool has(int q) const { return q == 0 ? rows > 0 : rows_1 > 0; }
};

}  // namespace ifx
