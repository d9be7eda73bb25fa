"""Decoded tokens with uneven numbers of keys: longest first, and in more parts than an even step would take, against float64."""
import math

import pytest
import torch

from tests.test_kernels_gpu import DEV, attention_oracle, fill_cache, make_cache_case, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nkv,page,longest,parts", [(8, 4, 16, 5700, 4), (4, 4, 32, 4100, 2), (8, 4, 16, 3900, 1)])
def test_uneven_decode(cuda_kernels, nq, nkv, page, longest, parts):
    n, d = 38, 128
    lens = [1 + 13 * i for i in range(n)]
    lens[5] = longest
    spans = [1] * n
    ctx, cache, slots = make_cache_case(torch.bfloat16, nkv, d, page, lens, spans, num_pages=sum(-(-k // page) for k in lens) + 3, seed=3)
    from inferflux_b200.csrc import CudaKernels
    meta = torch.tensor(CudaKernels.attention_sections(CudaKernels, ctx)["attn.decode_meta"]).view(n, 4)
    order = sorted(range(n), key=lambda r: -lens[r])
    assert meta[:, 0].tolist() == order and meta[:, 1].tolist() == [lens[r] - 1 for r in order]
    assert meta[:, 2].tolist() == [slots[r] for r in order]
    assert cuda_kernels.decode_splits(n, nkv, longest) == 1 and cuda_kernels.least_decode_splits(ctx, n, nkv, d, 0) == parts
    stored = fill_cache(cache, lens, slots, nkv, d, torch.bfloat16, seed=4)
    q = rnd(n, nq, d, dtype=torch.bfloat16, seed=5)
    scale = 1.0 / math.sqrt(d)
    want = attention_oracle(q, stored, lens, spans, nq, nkv, d, None, scale)
    got = cuda_kernels.attention(q.view(n, nq * d), nq, nkv, d, None, scale, ctx, cache).cpu().double()
    cuda_kernels.check_errors()
    # probabilities and results are rounded to bfloat16 (2^-8 of themselves at most)
    size = attention_oracle(q, [(k, v.abs()) for k, v in stored], lens, spans, nq, nkv, d, None, scale)
    assert ((got - want).abs() <= 1.1 * ((2 ** -8 + 1e-4) * size + 2 ** -8 * want.abs() + 1e-6)).all()
    # an even step keeps its one part
    ctx.spans = [(500, 1)] * n
    CudaKernels.attention_sections(CudaKernels, ctx)
    assert cuda_kernels.least_decode_splits(ctx, n, nkv, d, 0) == 1
