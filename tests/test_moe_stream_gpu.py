"""The experts of steps with few tokens on the tensor cores: token counts around the steps of the product's width, K and
outputs that fill no tile, experts without a token, one expert with all of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _inputs(T, width, ff, experts, outputs, top, glu, seed):
    g = torch.Generator().manual_seed(seed)
    h = torch.randn(T, width, generator=g).to(BF)
    up = (width ** -0.5 * torch.randn(experts, (2 if glu else 1) * ff, width, generator=g)).to(BF)
    down = (ff ** -0.5 * torch.randn(experts, width, ff, generator=g)).to(BF)
    ids = torch.stack([torch.randperm(outputs, generator=g)[:top] for _ in range(T)]).to(torch.int32)
    return h, up, down, ids, torch.rand(T, top, generator=g)


def _plain(h, up, down, ids, weights, experts, glu):
    """In 64 bits, with the activations rounded to bfloat16 where the kernels round them."""
    ff, out = down.shape[2], torch.zeros(h.shape, dtype=torch.float64)
    for t in range(h.shape[0]):
        for e, w in zip(ids[t].tolist(), weights[t].double()):
            if e >= experts:
                out[t] += w * h[t].double()
                continue
            z = up[e].double() @ h[t].double()
            if glu is None:
                act = z.clamp(min=0).square()
            else:
                gate, u = z[:ff].clamp(max=glu[0]), z[ff:].clamp(-glu[0], glu[0])
                act = gate * torch.sigmoid(glu[1] * gate) * (u + glu[2])
            out[t] += w * (down[e].double() @ act.to(BF).double())
    return out


@pytest.mark.parametrize("glu", [None, (7.0, 1.702, 1.0), (float("inf"), 1.0, 0.0)])
@pytest.mark.parametrize("T,width,ff,experts,identity,top", [
    (1, 64, 64, 4, 0, 2), (5, 72, 40, 5, 2, 3), (16, 136, 200, 3, 0, 3), (17, 256, 136, 6, 1, 2), (33, 64, 1032, 16, 0, 4),
    (65, 320, 72, 9, 0, 3), (127, 128, 96, 4, 0, 4), (300, 64, 72, 7, 1, 1),
    (1, 64, 72, 1024, 0, 2), (3, 72, 64, 33, 1, 4), (20, 64, 72, 300, 2, 3)])                    # fewer pairs than experts
def test_stream_against_64_bits(cuda_kernels, T, width, ff, experts, identity, top, glu):
    args = _inputs(T, width, ff, experts, experts + identity, top, glu, T + width)
    want = _plain(*args, experts, glu)
    h, up, down, ids, weights = (t.to(DEV) for t in args)
    for out_dtype in (torch.float32, BF):
        got = cuda_kernels._moe_experts_stream(h, up, down, ids, weights, experts, out_dtype, glu=glu)
        assert got.dtype == out_dtype
        # an activation may round to the neighbour of the 64-bit one (2^-8 of it), each on its own; and the result's rounding
        err = (got.double().cpu() - want).abs().max()
        assert float(err) <= (4 * 2.0 ** -8 * ff ** -0.5 + (0 if out_dtype == torch.float32 else 2.0 ** -8)) * max(1.0, float(want.abs().max()))
    cuda_kernels.check_errors()


def test_one_expert_takes_all_and_a_token_names_it_twice(cuda_kernels):
    """More pairs than a block takes at once, and other experts with none."""
    T, width, ff, experts = 160, 64, 72, 5
    h, up, down, ids, weights = _inputs(T, width, ff, experts, experts, 2, None, 1)
    ids[:] = 3
    want = _plain(h, up, down, ids, weights, experts, None)
    got = cuda_kernels._moe_experts_stream(h.to(DEV), up.to(DEV), down.to(DEV), ids.to(DEV), weights.to(DEV), experts, torch.float32)
    cuda_kernels.check_errors()
    assert float((got.double().cpu() - want).abs().max()) <= 4 * 2.0 ** -8 * ff ** -0.5 * max(1.0, float(want.abs().max()))


def test_a_token_that_is_not_finite_touches_no_other(cuda_kernels):
    T, width, ff, experts = 24, 128, 136, 4
    h, up, down, ids, weights = (t.to(DEV) for t in _inputs(T, width, ff, experts, experts, 2, None, 2))
    clean = cuda_kernels._moe_experts_stream(h, up, down, ids, weights, experts, BF)
    h[7, 3] = float("inf")
    h[9, 127] = float("nan")
    got = cuda_kernels._moe_experts_stream(h, up, down, ids, weights, experts, BF)
    keep = torch.ones(T, dtype=torch.bool, device=DEV)
    keep[7] = keep[9] = False
    assert torch.equal(got[keep], clean[keep])


@pytest.mark.parametrize("pairs,experts,width,ff,gated,want", [
    (4, 16, 64, 32, True, "tokens"), (4, 16, 1536, 2240, True, "stream"), (96, 16, 1536, 2240, True, "stream"),
    (188, 16, 1536, 2240, True, "stream"), (192, 16, 1536, 2240, True, "tiles"), (28, 16, 3584, 4736, True, "stream"),
    (32, 16, 3584, 4736, True, "tiles"), (300, 3, 64, 32, False, "tokens"), (520, 3, 64, 32, False, "tiles")])
def test_which_kernels_run(cuda_kernels, pairs, experts, width, ff, gated, want):
    assert cuda_kernels.moe_kernels(pairs, experts, width, ff, gated) == want


@pytest.mark.parametrize("pairs,experts,width,ff,gated,want", [
    (8, 64, 2048, 1408, True, "stream"), (24, 64, 2048, 1408, True, "stream"), (96, 64, 2048, 1408, True, "stream"),
    (300, 64, 2048, 1408, True, "stream"), (64, 256, 2048, 1024, True, "stream"), (192, 256, 2048, 1024, True, "stream"),
    (384, 256, 2048, 1024, True, "stream"), (511, 16, 2048, 1024, True, "tiles"), (200, 1025, 1024, 512, True, "tokens"),
    (512, 256, 2048, 1024, True, "tiles"),
    (1, 1024, 8000, 2500, False, "stream"), (1, 1024, 8000, 2499, False, "tokens"), (1, 1025, 8000, 2500, False, "tokens"),
    (511, 1024, 128, 128, True, "tokens"), (512, 1024, 128, 128, True, "tiles")])
def test_which_kernels_run_with_many_experts(cuda_kernels, pairs, experts, width, ff, gated, want):
    """From 40M multiply-adds or 512 pairs on over sorted rows, up to 1,024 experts below 512 pairs."""
    assert cuda_kernels.moe_kernels(pairs, experts, width, ff, gated) == want


@pytest.mark.parametrize("T,experts,ff", [(1, 4, 72), (2, 3, 1032), (255, 4, 72), (256, 4, 72), (60, 8, 640), (100, 8, 640)])
def test_the_rule_is_what_runs(cuda_kernels, T, experts, ff, monkeypatch):
    """Per token two launches, over sorted rows five; and the bits of the kernels that the rule names."""
    width, top = 256, 2
    monkeypatch.setattr(type(cuda_kernels), "MOE_TOKENS_MAX_WORK", 1_000_000)      # both sides of the line with small matrices
    for glu in (None, (7.0, 1.702, 1.0)):
        h, up, down, ids, weights = (t.to(DEV) for t in _inputs(T, width, ff, experts, experts, top, glu, T))
        way = cuda_kernels.moe_kernels(T * top, experts, width, ff, glu is not None)
        before = cuda_kernels.launches
        got = cuda_kernels.moe_experts(h, up, down, ids, weights, experts, BF, glu=glu)
        assert cuda_kernels.launches - before == (2 if way == "tokens" else 5)
        if way != "tokens":
            by = cuda_kernels._moe_experts_stream if way == "stream" else cuda_kernels._moe_experts_tiles
            assert torch.equal(got, by(h, up, down, ids, weights, experts, BF, glu=glu))
        assert way == {(1, 72): "tokens", (2, 1032): "stream", (255, 72): "tiles", (256, 72): "tiles", (60, 640): "stream",
                       (100, 640): "tiles"}[T, ff]
    cuda_kernels.check_errors()


def test_more_experts_than_the_stream_and_the_tiles_take(cuda_kernels):
    """Between 192 and 511 pairs they go per token."""
    T, width, ff, experts = 100, 64, 72, 1100
    h, up, down, ids, weights = _inputs(T, width, ff, experts, experts, 2, None, 3)
    want = _plain(h, up, down, ids, weights, experts, None)
    got = cuda_kernels.moe_experts(h.to(DEV), up.to(DEV), down.to(DEV), ids.to(DEV), weights.to(DEV), experts, torch.float32)
    assert float((got.double().cpu() - want).abs().max()) <= 4 * 2.0 ** -8 * ff ** -0.5 * max(1.0, float(want.abs().max()))
