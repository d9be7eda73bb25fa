"""Prompt attention of more blocks than SMs: a resident block that goes through several blocks of the grid gives every one of them
the bits it has in a grid of its own."""
import math
import random

import pytest
import torch

from tests.test_kernels_gpu import DEV, _Ctx, fill_cache, make_cache_case

pytestmark = pytest.mark.gpu

LENS = [1024, 130, 1003, 5, 640, 300, 900, 129, 1024, 257, 512]
SPANS = [256, 130, 1000, 5, 128, 300, 1, 129, 2, 257, 131]          # one and two query tiles, one row of a second, a decoded token


def _alone(ctx, r):
    from inferflux_b200.csrc import CudaKernels
    one, first = _Ctx(), sum(n for _s, n in ctx.spans[:r])
    one.spans, one.slots_host = [ctx.spans[r]], [ctx.slots_host[r]]
    one.num_tokens = ctx.spans[r][1]
    one.positions = ctx.positions[first:first + one.num_tokens].clone()
    one.token_req = torch.zeros(one.num_tokens, dtype=torch.int32, device=DEV)
    one.req_slot = ctx.req_slot[r:r + 1].clone()
    one.extra, one.extra_len = {}, {}
    for name, vals in CudaKernels.attention_sections(CudaKernels, one).items():
        one.extra[name] = torch.tensor(vals, dtype=torch.int32, device=DEV)
        one.extra_len[name] = len(vals)
    one.max_kv_len = sum(ctx.spans[r])
    return one, slice(first, first + one.num_tokens)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window,keep", [(None, 0), (200, 0), (200, 300)])
def test_blocks_behind_one_another(cuda_kernels, d, window, keep):
    nq, nkv, page = 36, 4, 16
    ctx, cache, slots = make_cache_case(torch.bfloat16, nkv, d, page, LENS, SPANS, num_pages=sum(-(-n // page) for n in LENS) + 3, seed=3)
    fill_cache(cache, LENS, slots, nkv, d, torch.bfloat16, seed=4)
    blocks = ctx.extra_len["attn.prefill_tiles"] // 4 * nq
    assert blocks > 3 * 148 and cuda_kernels.prefill_parts(ctx, nq, window or 0) == 1
    q = torch.randn(ctx.num_tokens, nq * d, generator=torch.Generator().manual_seed(5)).bfloat16().to(DEV)
    args = (nq, nkv, d, window, 2.0 / math.sqrt(d))
    got = [cuda_kernels.attention(q, *args, ctx, cache, keep_first=keep) for _ in range(3)]
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])          # whichever SM takes which block
    for r, span in enumerate(SPANS):
        one, rows = _alone(ctx, r)
        assert one.extra_len["attn.prefill_tiles"] // 4 * nq <= 148
        want = cuda_kernels.attention(q[rows].contiguous(), *args, one, cache, keep_first=keep)
        if span > 1:
            assert torch.equal(got[0][rows], want), r
        else:                                       # (a decoded token's keys are cut by how many tokens there are)
            assert (got[0][rows].float() - want.float()).abs().max() <= 2 ** -6
    cuda_kernels.check_errors()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [None, 200])
@pytest.mark.parametrize("lens,spans", [([300], [257]), ([128, 129, 700, 5], [128, 129, 130, 1]), ([1000], [1000]), ([60, 256], [60, 256])])
def test_a_block_for_each_128_rows(cuda_kernels, monkeypatch, d, window, lens, spans):
    """The same bits as with 256 rows a block; second query tiles that are there, of one row, and not there."""
    nq, nkv, page = 12, 4, 16
    ctx, cache, slots = make_cache_case(torch.bfloat16, nkv, d, page, lens, spans, num_pages=sum(-(-n // page) for n in lens) + 3, seed=3)
    fill_cache(cache, lens, slots, nkv, d, torch.bfloat16, seed=4)
    assert cuda_kernels.prefill_parts(ctx, nq, window or 0) == 1 and cuda_kernels.prefill_cut(ctx, nq, window or 0) == -1
    q = torch.randn(ctx.num_tokens, nq * d, generator=torch.Generator().manual_seed(5)).bfloat16().to(DEV)
    args = (nq, nkv, d, window, 2.0 / math.sqrt(d), ctx, cache)
    got = cuda_kernels.attention(q, *args)
    monkeypatch.setattr(type(cuda_kernels), "_prefill_by_tiles", staticmethod(lambda ctx, nq: False))
    ctx.__dict__.pop("prefill_parts")
    assert cuda_kernels.prefill_cut(ctx, nq, window or 0) == 1
    assert torch.equal(got, cuda_kernels.attention(q, *args))
    cuda_kernels.check_errors()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [None, 200])
def test_blocks_of_one_query_tile_behind_one_another(cuda_kernels, d, window):
    """Many rounds of blocks without a second query tile (whose softmax group only reads which block is next), a few with one between them."""
    nq, nkv, page = 36, 4, 16
    r = random.Random(7)
    spans = [256 if i % 23 == 5 else 130 if i % 23 == 6 else r.randint(2, 128) for i in range(92)]
    lens = [n + r.choice([0, 0, 30, 500]) for n in spans]
    ctx, cache, slots = make_cache_case(torch.bfloat16, nkv, d, page, lens, spans, num_pages=sum(-(-n // page) for n in lens) + 3, seed=3)
    fill_cache(cache, lens, slots, nkv, d, torch.bfloat16, seed=4)
    assert ctx.extra_len["attn.prefill_tiles"] // 4 * nq > 20 * 148
    q = torch.randn(ctx.num_tokens, nq * d, generator=torch.Generator().manual_seed(5)).bfloat16().to(DEV)
    args = (nq, nkv, d, window, 2.0 / math.sqrt(d))
    got = [cuda_kernels.attention(q, *args, ctx, cache) for _ in range(5)]
    assert all(torch.equal(g, got[0]) for g in got)
    for i in range(0, len(spans), 5):
        one, rows = _alone(ctx, i)
        assert torch.equal(got[0][rows], cuda_kernels.attention(q[rows].contiguous(), *args, one, cache)), i
    cuda_kernels.check_errors()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [None, 60, 200])
@pytest.mark.parametrize("lens,spans", [([700] * 12, [100] * 12), ([128 + 3 * i for i in range(40)], [2 + 3 * i for i in range(40)]),
                                        ([900, 300, 400], [256, 1 + 128, 100])])
def test_second_query_tiles_that_are_not_there(cuda_kernels, monkeypatch, d, window, lens, spans):
    """A block for each 128 rows in grids of more blocks than SMs, items of 128 rows and fewer behind more keys than a window holds."""
    nq, nkv, page = 24, 4, 16
    ctx, cache, slots = make_cache_case(torch.bfloat16, nkv, d, page, lens, spans, num_pages=sum(-(-n // page) for n in lens) + 3, seed=3)
    fill_cache(cache, lens, slots, nkv, d, torch.bfloat16, seed=4)
    monkeypatch.setattr(cuda_kernels, "prefill_parts", lambda *a: 1)
    q = torch.randn(ctx.num_tokens, nq * d, generator=torch.Generator().manual_seed(5)).bfloat16().to(DEV)
    results = []
    for by_tiles in (True, False):
        ctx.__dict__.pop("prefill_parts", None)
        monkeypatch.setattr(type(cuda_kernels), "_prefill_by_tiles", staticmethod(lambda ctx, nq: by_tiles))
        assert cuda_kernels.prefill_cut(ctx, nq, window or 0) == (-1 if by_tiles else 1)
        results += [cuda_kernels.attention(q, nq, nkv, d, window, 2.0 / math.sqrt(d), ctx, cache) for _ in range(3)]
    assert all(torch.equal(g, results[0]) for g in results)
    cuda_kernels.check_errors()
