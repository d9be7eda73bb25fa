"""The experts over sorted rows, products by pairs of SMs: pairs of an expert around the tiles' widths (16, 32, 256 rows), matrices
that fill no tile of 128 or 256 outputs or 64 of K, experts without a pair, one with all of them, experts without weights."""
import math

import pytest
import torch
from test_moe_stream_gpu import BF, DEV, _inputs, _plain

pytestmark = pytest.mark.gpu


def _bound(want, ff, out_dtype):
    """An activation may round to the neighbour of the 64-bit one (2^-8 of it), each on its own; and the result's rounding."""
    return (4 * 2.0 ** -8 * ff ** -0.5 + (0 if out_dtype == torch.float32 else 2.0 ** -8)) * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("glu", [None, (7.0, 1.702, 1.0), (float("inf"), 1.0, 0.0)])
@pytest.mark.parametrize("T,width,ff,experts,identity,top", [
    (1, 64, 64, 4, 0, 1), (16, 72, 40, 2, 0, 2), (33, 136, 200, 3, 2, 3), (97, 256, 136, 6, 1, 2), (255, 64, 264, 1, 0, 1),
    (256, 320, 72, 1, 0, 1), (257, 264, 128, 2, 0, 2), (600, 64, 392, 5, 1, 4), (40, 72, 64, 1000, 3, 4), (3, 520, 1032, 300, 0, 3)])
def test_against_64_bits(cuda_kernels, T, width, ff, experts, identity, top, glu):
    args = _inputs(T, width, ff, experts, experts + identity, top, glu, T + width)
    want = _plain(*args, experts, glu)
    h, up, down, ids, weights = (t.to(DEV) for t in args)
    for out_dtype in (torch.float32, BF):
        got = cuda_kernels._moe_experts_tiles(h, up, down, ids, weights, experts, out_dtype, glu=glu)
        assert got.dtype == out_dtype
        assert float((got.double().cpu() - want).abs().max()) <= _bound(want, ff, out_dtype)
    cuda_kernels.check_errors()


@pytest.mark.parametrize("T", [31, 32, 33, 255, 257, 513])
def test_one_expert_takes_all_and_others_few(cuda_kernels, T):
    width, ff, experts = 136, 264, 5
    h, up, down, ids, weights = _inputs(T, width, ff, experts, experts, 2, None, T)
    ids[:], ids[T // 2, 1] = 3, 0
    want = _plain(h, up, down, ids, weights, experts, None)
    got = cuda_kernels._moe_experts_tiles(h.to(DEV), up.to(DEV), down.to(DEV), ids.to(DEV), weights.to(DEV), experts, torch.float32)
    cuda_kernels.check_errors()
    assert float((got.double().cpu() - want).abs().max()) <= _bound(want, ff, torch.float32)


def test_rows_that_are_no_numbers_stay_alone(cuda_kernels):
    """A token's infinities and NaN reach its own result and no other token's, whatever tile they share."""
    T, width, ff, experts = 300, 128, 144, 3
    glu = (7.0, 1.702, 1.0)
    h, up, down, ids, weights = (t.to(DEV) for t in _inputs(T, width, ff, experts, experts, 2, glu, 5))
    clean = cuda_kernels._moe_experts_tiles(h, up, down, ids, weights, experts, BF, glu=glu)
    h[7, 3], h[100, 0] = float("inf"), float("nan")
    got = cuda_kernels._moe_experts_tiles(h, up, down, ids, weights, experts, BF, glu=glu)
    keep = torch.ones(T, dtype=torch.bool, device=DEV)
    keep[[7, 100]] = False
    assert torch.equal(got[keep], clean[keep])


@pytest.mark.parametrize("T,width,ff,slices", [(5, 64, 704, 1), (3, 64, 712, 3), (40, 136, 768, 3), (33, 72, 840, 3)])
def test_few_tokens_add_slices_of_the_second_product_in_float32(cuda_kernels, T, width, ff, slices):
    """Bit for bit: a slice is the same product over a part of the inner size; weighted, then added, each step rounded."""
    experts, top = 4, 2
    h, up, down, ids, weights = (t.to(DEV) for t in _inputs(T, width, ff, experts, experts + 1, top, None, T))
    per = -(-(-(-ff // 64)) // slices) * 64
    parts = []
    for k in range(0, ff, per):
        w_up, w_down = up[:, k:k + per].contiguous(), down[:, :, k:k + per].contiguous()
        parts.append([cuda_kernels._moe_experts_tiles(h, w_up, w_down, ids[:, c:c + 1].contiguous(), torch.ones(T, 1, device=DEV), experts,
                                                      torch.float32) for c in range(top)])
    assert len(parts) == slices
    want = torch.zeros(T, width, device=DEV)
    for c in range(top):
        w = weights[:, c:c + 1]
        sums = want
        for part in parts:
            sums = sums + part[c] * w
        plain = torch.addcmul(want, w, h.float())                            # an expert without weights
        want = torch.where(ids[:, c:c + 1] < experts, sums, plain)
    for out_dtype in (torch.float32, BF):
        got = cuda_kernels._moe_experts_stream(h, up, down, ids, weights, experts, out_dtype)
        assert torch.equal(got, want.to(out_dtype))
    cuda_kernels.check_errors()


def test_gates_of_few_tokens_are_divided_exactly(cuda_kernels):
    """silu(-88) is 5e-37, which a fast division by 1 + e^88 takes for 0."""
    experts, width, ff = 2, 64, 64
    h, up, down = torch.zeros(3, width), torch.zeros(experts, 2 * ff, width), torch.zeros(experts, width, ff)
    h[:, 0], up[:, :ff, 0], up[:, ff:, 0], down[:, :, 5] = 1.0, -88.0, 1.0, 2.0 ** 100
    ids, weights = torch.zeros(3, 1, dtype=torch.int32, device=DEV), torch.ones(3, 1, device=DEV)
    got = cuda_kernels._moe_experts_stream(h.to(BF).to(DEV), up.to(BF).to(DEV), down.to(BF).to(DEV), ids, weights, experts, torch.float32,
                                           glu=(float("inf"), 1.0, 0.0))
    want = -88.0 * math.exp(-88.0) * 2.0 ** 100
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * abs(want)).all())
