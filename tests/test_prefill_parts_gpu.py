"""Prompt attention whose left over blocks are cut into parts of their keys, against float64."""
import math

import pytest
import torch

from tests.test_kernels_gpu import DEV, fill_cache, make_cache_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nkv,d,page,window,lens,spans,parts", [
    (12, 2, 128, 16, None, [1400], [300], 2),                     # 24 blocks, all of them cut; a second query tile of 44 rows
    (4, 2, 64, 16, None, [3200, 40, 700], [130, 1, 2], 6),        # another request's few keys behind a long one; empty parts
    (28, 4, 128, 16, None, [2100], [1537], 2),                    # 196 blocks: a whole round and 48 left over
    (6, 1, 128, 32, 900, [2500], [256], 2),                       # a window: parts in front of its rows' first keys
    (6, 1, 64, 16, None, [1153], [257], 2)])                      # the last item is one row
def test_parts_of_keys(cuda_kernels, nq, nkv, d, page, window, lens, spans, parts):
    ctx, cache, slots = make_cache_case(torch.bfloat16, nkv, d, page, lens, spans, num_pages=sum(-(-n // page) for n in lens) + 3, seed=3)
    stored = fill_cache(cache, lens, slots, nkv, d, torch.bfloat16, seed=4)
    T = ctx.num_tokens
    g = torch.Generator().manual_seed(5)
    q = torch.randn(T, nq, d, generator=g).bfloat16()
    scale = 2.0 / math.sqrt(d)
    assert cuda_kernels.prefill_parts(ctx, nq, window or 0) == parts
    before = cuda_kernels.launches
    got = cuda_kernels.attention(q.to(DEV).view(T, nq * d), nq, nkv, d, window, scale, ctx, cache).cpu().double().view(T, nq, d)
    assert cuda_kernels.launches - before == 2 + any(s == 1 for s in spans)
    cuda_kernels.check_errors()
    t = 0
    for (K, V), n, s in zip(stored, lens, spans):
        pos = torch.arange(n - s, n)[:, None]
        key = torch.arange(n)[None]
        seen = (key <= pos) & ((key > pos - window) if window else torch.ones_like(key, dtype=torch.bool))
        for h in range(nq):
            k, v = K[:, h // (nq // nkv)].double(), V[:, h // (nq // nkv)].double()
            p = torch.softmax((q[t:t + s, h].double() @ k.T * scale).masked_fill(~seen, -torch.inf), -1)
            want, size = p @ v, p @ v.abs()
            # probabilities and results are rounded to bfloat16 (2^-8 of themselves at most, half a spacing); float32 sums of up to n terms otherwise
            bound = (2 ** -8 + 1e-4) * size + 2 ** -8 * want.abs() + 1e-6
            assert ((got[t:t + s, h] - want).abs() <= 1.1 * bound).all(), (h, t)
        t += s


def test_bytes_of_the_parts(cuda_kernels):
    for case in ((2, 12, 128, 2), (7, 28, 128, 2), (1, 4, 64, 6), (37, 4, 64, 3)):
        assert cuda_kernels.prefill_parts_bytes(*case) == cuda_kernels.lib.ifx_attention_prefill_tcgen05_parts_bytes(*case)
