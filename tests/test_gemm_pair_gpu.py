"""Products by pairs of SMs with one matrix: rows around the tiles' sizes, outputs and K that fill no tile, outputs in eights and
sixteens (gate and up rows lie interleaved by the larger that fits), rows that are no numbers."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _operands(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    return (0.5 * torch.randn(M, K, generator=g)).to(BF).to(DEV), (0.1 * torch.randn(2 * N, K, generator=g)).to(BF).to(DEV)


# 70 and 150 tiles of outputs: less and more than a wave of pairs
@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (31, 24, 72), (33, 136, 8), (161, 264, 200), (256, 128, 64), (257, 1000, 136), (511, 40, 1536),
                                   (1025, 392, 264), (300, 8960, 264), (530, 19208, 72)])
def test_against_64_bits(cuda_kernels, M, N, K):
    a, w = _operands(M, N, K)
    z = a.double() @ w.double().t()
    g, u = z[:, :N], z[:, N:]
    # the sums' float32 additions (2^-23 of the products' sizes a K step of the tensor cores at most), then the rounding to bfloat16
    tol = 1e-4 * math.sqrt(K)
    got, want = cuda_kernels.linear_tiles(a, w, swiglu=True).double(), g * torch.sigmoid(g) * u
    assert bool(((got - want).abs() <= tol + 2.0 ** -7 * want.abs()).all())
    if M > cuda_kernels.SKINNY_MAX_ROWS:
        got, want = cuda_kernels.linear_relu2(a, w[:N].contiguous()).double(), g.clamp(min=0).square()
        assert bool(((got - want).abs() <= tol + 2.0 ** -7 * want.abs()).all())
    cuda_kernels.check_errors()


def test_rows_that_are_no_numbers_stay_alone(cuda_kernels):
    a, w = _operands(300, 264, 72)
    clean = cuda_kernels.linear_tiles(a, w, swiglu=True)
    a[5, 3], a[299, 0] = float("nan"), float("inf")
    got = cuda_kernels.linear_tiles(a, w, swiglu=True)
    keep = torch.ones(300, dtype=torch.bool, device=DEV)
    keep[[5, 299]] = False
    assert torch.equal(got[keep], clean[keep]) and bool(got[5].isnan().all()) and not bool(got[299].isfinite().any(dim=0).all())
