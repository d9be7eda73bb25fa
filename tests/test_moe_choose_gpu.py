"""Router and choice in one launch against the logits in 64 bits and the choice from given logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("kind", [{}, {"of_chosen": True}, {"kind": "sigmoid_normalized", "floor": 1e-20}])
@pytest.mark.parametrize("T,K,n,top", [(1, 8, 1, 1), (5, 40, 8, 3), (16, 1536, 16, 4), (17, 776, 9, 2), (33, 1528, 18, 4), (300, 3584, 24, 6),
                                       (100, 256, 25, 4), (40, 2048, 33, 8), (24, 1536, 64, 4), (19, 512, 64, 40),
                                       (20, 512, 40, 32)])
def test_router_and_choice(cuda_kernels, kind, T, K, n, top):
    g = torch.Generator().manual_seed(T * K + n)
    h = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w = (K ** -0.5 * torch.randn(n, K, generator=g)).to(torch.bfloat16)
    corr = None if kind.get("of_chosen") else 0.1 * torch.randn(n, generator=g).to(DEV)
    ids, weights = cuda_kernels.moe_choose(h.to(DEV), w.to(DEV), corr, top, **kind)
    z = (h.double() @ w.double().T)
    want_ids, want = cuda_kernels.moe_route(z.float().to(DEV), corr, top, **kind)
    same = (ids == want_ids).all(1)
    assert float(same.float().mean()) > 0.98                 # (logits a rounding apart may change places)
    # logits are float32 sums of K products: good to about sqrt(K) roundings of their size, weights of them alike
    assert float((weights - want)[same].abs().max()) <= 4e-6
    # a token's choice depends on nothing else in the step, to the bit
    lone = cuda_kernels.moe_choose(h[T - 1:].to(DEV), w.to(DEV), corr, top, **kind)
    assert torch.equal(lone[0][0], ids[-1]) and torch.equal(lone[1][0], weights[-1])


def test_wide_or_misaligned_routers_take_two_launches(cuda_kernels):
    g = torch.Generator().manual_seed(5)
    for K, n, off in ((64, 65, 0), (64, 16, 1), (60, 16, 0)):
        h = torch.randn(3, K, generator=g).to(torch.bfloat16).to(DEV)
        w = torch.empty(n * K + off, dtype=torch.bfloat16, device=DEV)[off:].view(n, K).copy_(torch.randn(n, K, generator=g))
        got = cuda_kernels.moe_choose(h, w, None, 2, of_chosen=True)
        want = cuda_kernels.moe_route(cuda_kernels.linear(h, w, out_dtype=torch.float32), None, 2, of_chosen=True)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("kind", [{}, {"of_chosen": True}, {"kind": "sigmoid_normalized", "floor": 1e-20}])
@pytest.mark.parametrize("n", [5, 32, 47])
def test_ties_and_logits_that_are_not_finite(cuda_kernels, kind, n):
    """One-hot rows hand chosen logits through exactly: equal ones, zeros of both signs, infinities and NaN choose as given logits do."""
    g = torch.Generator().manual_seed(n)
    z = torch.randint(-2, 3, (40, n), generator=g).float()
    z[1, 2], z[2, :] = -0.0, 0.0
    z[3, 0], z[3, 1] = float("inf"), float("-inf")
    z[4, :3] = float("-inf")
    K = 48
    h = torch.zeros(40, K)
    h[:, :40] = torch.eye(40)
    w = torch.zeros(n, K)
    w[:, :40] = z.T
    finite = torch.isfinite(z).all(1)
    w = torch.nan_to_num(w, posinf=0.0, neginf=0.0)          # (an infinite weight would meet every other row's zeros)
    corr = None if kind.get("of_chosen") else torch.zeros(n).to(DEV)
    got = cuda_kernels.moe_choose(h.to(torch.bfloat16).to(DEV), w.to(torch.bfloat16).to(DEV), corr, 4, **kind)
    want = cuda_kernels.moe_route((h @ w.T).to(DEV), corr, 4, **kind)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    for i in (~finite).nonzero()[:, 0].tolist() + [0]:       # one row alone, whose logits are what the weights say
        col = z[i:i + 1].T.clone()
        if i == 0:
            col[1], col[3] = float("nan"), float("nan")
        one = torch.zeros(1, 8, dtype=torch.bfloat16)
        one[0, 0] = 1
        wide = torch.zeros(n, 8)
        wide[:, :1] = col
        got = cuda_kernels.moe_choose(one.to(DEV), wide.to(torch.bfloat16).to(DEV), corr, 2, **kind)
        want = cuda_kernels.moe_route(col.T.contiguous().to(DEV), corr, 2, **kind)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1].isnan(), want[1].isnan())
        assert torch.equal(got[1].nan_to_num(), want[1].nan_to_num())
