"""What the blocks of prompt attention walk (prefill_item.cuh, compiled for the host): every key tile that a block fetches is used by one of
its query tiles, no page beyond a request's keys is looked up, and together the blocks see every key of every row once."""
import ctypes
import importlib
import random
import shutil
import subprocess

import pytest

build = importlib.import_module("inferflux_b200.csrc.build")
SOURCE = r"""
#include "prefill_item.cuh"
using namespace ifx;
template <bool KEPT>
static int walk(const int* tiles, int num_tiles, int nq, int block, KeyMask mask, PrefillParts split, int* about, int* out) {
  const PrefillItem<KEPT> it(block, tiles, num_tiles, nq, mask, split);
  const int known[] = {it.r, it.row0, it.rows, it.rows_1, it.pos0, it.h, it.slot, it.visits(), it.has(0), it.has(1)};
  for (int i = 0; i < 10; ++i) about[i] = known[i];
  int n = 0;
  for (int kt = it.tb; kt < it.te && n < 1000; kt = it.next_tile(kt), ++n) {
    out[4 * n] = kt, out[4 * n + 1] = it.visited(kt), out[4 * n + 2] = it.active(0, kt), out[4 * n + 3] = it.active(1, kt);
  }
  return n;
}
extern "C" int walk_block(const int* tiles, int num_tiles, int nq, int block, int window, int chunk, int keep, int full, int parts, int halves,
                          int* about, int* out) {
  const KeyMask mask{window, chunk, 0, nullptr, keep};
  const PrefillParts split{full, parts, halves, nullptr, nullptr};
  return keep > 0 ? walk<true>(tiles, num_tiles, nq, block, mask, split, about, out) : walk<false>(tiles, num_tiles, nq, block, mask, split, about, out);
}
"""


@pytest.fixture(scope="module")
def walk_block(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("prefill_items")
    (d / "walk.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-x", "c++", "-std=c++17", "-shared", "-fPIC", "-O1", "-I", str(build.HERE), str(d / "walk.cpp"), "-o", str(d / "walk.so")],
                   check=True)
    return ctypes.CDLL(str(d / "walk.so")).walk_block


def _first(pos, window, chunk):
    return max(pos - window + 1 if window else 0, pos // chunk * chunk if chunk else 0, 0)


def _check(walk_block, spans, nq, window, chunk, keep, parts):
    tiles, row = [], 0                                       # as CudaKernels.attention_sections lays them out: 256 rows an item
    for r, (s, n) in enumerate(spans):
        for t in range(0, n, 256):
            tiles.append((r, row + t, min(256, n - t), s + t))
        row += n
    blocks = len(tiles) * nq
    left = blocks % 148 if parts > 1 else 0
    full = 2 * blocks if parts == -1 else blocks - left
    flat = (ctypes.c_int * (4 * len(tiles)))(*[v for t in tiles for v in t])
    about, out = (ctypes.c_int * 10)(), (ctypes.c_int * 4000)()
    seen = {}                                                # (row tile, head): key tiles
    for block in range(full + left * max(parts, 1)):
        n = walk_block(flat, len(tiles), nq, block, window, chunk, keep, full, parts, int(parts == -1), about, out)
        r, row0, rows, rows_1, pos0, h, slot, visits, has0, has1 = about
        assert n == visits and (has0 or n == 0)
        last = sum(spans[r]) - 1
        first = _first(pos0, window, chunk)
        for i in range(n):
            kt, at, q0, q1 = out[4 * i:4 * i + 4]
            assert at == i and (q0 or q1), "a tile that no query uses"
            assert (has0 or not q0) and (has1 or not q1)
            for key in range(kt * 128, kt * 128 + 128, 16):  # the fetching warp's lanes
                assert not (key < pos0 + rows and (key + 16 > first or key < keep)) or key <= last, "a page beyond the request's keys"
            for q, used in ((0, q0), (1, q1)):
                if used:
                    seen.setdefault((row0 + 128 * q, h), []).append(kt)
    for r, row0, rows, pos in tiles:
        for q in range(-(-rows // 128)):
            a, b = pos + 128 * q, pos + min(rows, 128 * q + 128) - 1
            need = {k // 128 for p in range(a, b + 1) for k in (_first(p, window, chunk), p)}
            need |= set(range(min(need), max(need) + 1)) | {k // 128 for k in range(0, min(keep, b + 1), 128)}
            for h in range(nq):
                got = seen.pop((row0 + 128 * q, h))
                assert len(got) == len(set(got)) and need <= set(got)
    assert not seen


@pytest.mark.parametrize("parts", [1, 2, 5, -1])
@pytest.mark.parametrize("seed", range(6))
def test_every_tile_is_used(walk_block, parts, seed):
    r = random.Random(seed)
    for _ in range(12):
        spans = [(r.choice([0, 0, 3, 43, 100, 128, 256, 600, 700, 1500]), r.choice([2, 100, 127, 128, 129, 255, 256, 257, 300, 384, 385, 520]))
                 for _ in range(r.randint(1, 4))]
        window, chunk = r.choice([0, 1, 17, 100, 127, 128, 129, 200, 640]), r.choice([0, 0, 64, 200])
        _check(walk_block, spans, r.choice([1, 3]), window, chunk, r.choice([0, 5, 300]) if parts == 1 else 0, parts)


def test_short_items_far_behind_a_window(walk_block):
    """Second query tiles that are not there, at positions where a window has moved on."""
    _check(walk_block, [(43, 257)], 12, 200, 0, 0, -1)
    _check(walk_block, [(600, 100)] * 12, 12, 200, 0, 0, -1)
    for s in range(0, 700, 37):
        for window in (1, 64, 128, 200, 513):
            _check(walk_block, [(s, 1 + s % 128)], 1, window, 0, 0, -1)
