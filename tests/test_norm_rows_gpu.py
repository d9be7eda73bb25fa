"""RMS norms at the line between blocks for few rows and for many, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("hidden", [512, 520, 1536, 3584, 8192])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("add", [False, True])
def test_blocks_for_few_and_for_many_rows(cuda_kernels, hidden, more, add):
    rows = -(-1300000 // hidden) - 1 + more                             # the last of the one kind, the first of the other
    g = torch.Generator().manual_seed(hidden + more)
    x, w = torch.randn(rows, hidden, generator=g) * 3, torch.randn(hidden, generator=g)
    delta = torch.randn(rows, hidden, generator=g).bfloat16()
    stream = x.to(DEV)
    if add:
        got = cuda_kernels.add_rmsnorm(stream, delta.to(DEV), w.to(DEV), 1e-6, torch.bfloat16)
        x = x + delta.float()
        assert torch.equal(stream.cpu(), x)
    else:
        got = cuda_kernels.rmsnorm(stream, w.to(DEV), 1e-6, torch.bfloat16)
    # a row's bits do not depend on how many rows there are
    few = (cuda_kernels.add_rmsnorm(x[:9].to(DEV), torch.zeros(9, hidden).bfloat16().to(DEV), w.to(DEV), 1e-6, torch.bfloat16) if add
           else cuda_kernels.rmsnorm(x[:9].to(DEV), w.to(DEV), 1e-6, torch.bfloat16))
    assert torch.equal(few, got[:9])
    want = x.double() / (x.double().pow(2).mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
    # the result is rounded to bfloat16 (at most 2^-8 of itself); float32 sums of at most 8,192 squares and three products otherwise
    assert ((got.cpu().double() - want).abs() <= (2 ** -8 + 2e-6) * want.abs() + 1e-30).all()
