"""The float32 product's tiles at their edges: one row to several tiles of rows, columns and K that fill no tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K", [(1, 64, 4), (1, 1000, 1536), (8, 63, 68), (9, 9473, 36), (9, 200, 64), (16, 9472, 96), (17, 33, 132),
                                   (31, 4000, 100), (32, 65, 32), (33, 7700, 72), (65, 257, 1028), (333, 1536, 320)])
def test_tiles_make_the_bits_of_the_general_kernel(cuda_kernels, M, N, K):
    """An output is one chain of multiply-adds, k ascending, in both: operands off a 16-byte boundary take the general kernel."""
    g = torch.Generator().manual_seed(M * 7 + N + K)
    a, w, bias = (torch.randn(n, generator=g).to(DEV) for n in ((M, K), (N, K), (N,)))
    apart = [torch.empty(t.numel() + 1, device=DEV)[1:].view(t.shape).copy_(t) for t in (a, w)]
    assert apart[0].data_ptr() % 16 and a.data_ptr() % 16 == 0
    for b in (None, bias):
        assert torch.equal(cuda_kernels.linear(a, w, b), cuda_kernels.linear(*apart, b))
    want = a.double() @ w.double().t()
    # each of the K roundings is at most 2^-24 of a partial sum, which stays below the sum of the products' sizes
    bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 1e-30
    assert bool(((cuda_kernels.linear(a, w).double() - want).abs() <= bound).all())


def test_rows_do_not_depend_on_their_number(cuda_kernels):
    g = torch.Generator().manual_seed(3)
    a, w = torch.randn(200, 516, generator=g).to(DEV), torch.randn(700, 516, generator=g).to(DEV)
    whole = cuda_kernels.linear(a, w)
    for n in (1, 8, 9, 16, 17, 40, 130):
        assert torch.equal(cuda_kernels.linear(a[:n].contiguous(), w), whole[:n])
    a[5, 7] = float("inf")
    a[6, 515] = float("nan")
    got = cuda_kernels.linear(a, w)
    keep = torch.ones(200, dtype=torch.bool, device=DEV)
    keep[5:7] = False
    assert torch.equal(got[keep], whole[keep]) and not bool(torch.isfinite(got[5:7]).any())
