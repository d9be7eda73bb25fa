"""The feed-forward of few rows whose two products are launched by one call: the bits and the kind of result of the two calls that it
stands for, at the row counts where the second product's slices and the kernels change."""
import pytest
import torch

from inferflux_b200.csrc import PartialSum, ScaledRows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16
SIZES = {"slices": (256, 1032, 136), "one slice": (136, 72, 264), "a wave of tiles": (64, 264, 19000)}       # inner sizes, outputs


def _operands(T, K, inter, N):
    g = torch.Generator().manual_seed(T + K + N)
    make = lambda *s: (0.1 * torch.randn(*s, generator=g)).to(BF).to(DEV)
    return make(T, K), make(2 * inter, K), make(N, inter)


def _scaled(a, seed):
    g = torch.Generator().manual_seed(seed)
    return ScaledRows(a, (a.shape[1] / 3 * (0.5 + torch.rand(a.shape[0], 3, generator=g))).to(DEV), 1e-6)


@pytest.mark.parametrize("sizes", list(SIZES))
@pytest.mark.parametrize("T", [1, 16, 17, 128, 129, 160])
@pytest.mark.parametrize("scaled", [False, True])
def test_the_same_as_two_calls(cuda_kernels, T, sizes, scaled):
    assert cuda_kernels.SKINNY_MAX_ROWS == 160
    a, w_gate_up, w_down = _operands(T, *SIZES[sizes])
    rows = _scaled(a, T) if scaled else a
    got = cuda_kernels.swiglu_few(rows, w_gate_up, w_down)
    want = cuda_kernels.linear(cuda_kernels.linear_swiglu(rows, w_gate_up), w_down, allow_partial=True)
    assert type(got) is type(want) and isinstance(got, PartialSum) == (sizes == "slices")
    if isinstance(want, PartialSum):
        assert got.dtype == want.dtype and torch.equal(got.parts, want.parts)
    else:
        assert got.dtype == want.dtype and torch.equal(got, want)
    cuda_kernels.check_errors()


def test_what_it_leaves_to_the_others(cuda_kernels):
    K, inter, N = 136, 72, 264
    a, w_gate_up, w_down = _operands(161, K, inter, N)
    few = cuda_kernels.swiglu_few
    assert few(a, w_gate_up, w_down) is None and few(_scaled(a, 0), w_gate_up, w_down) is None
    assert few(a[:0], w_gate_up, w_down) is None
    a = a[:8].contiguous()
    assert few(a, w_gate_up, w_down) is not None
    assert few(a.float(), w_gate_up.float(), w_down.float()) is None and few(a, w_gate_up, w_down.float()) is None
    assert few(a.t().contiguous().t(), w_gate_up, w_down) is None
    assert few(a, w_gate_up[:, :128].contiguous(), w_down) is None and few(a, w_gate_up[:-8], w_down) is None
    shifted = torch.empty(8 * K + 1, dtype=BF, device=DEV)[1:].view(8, K)
    assert few(shifted, w_gate_up, w_down) is None
    odd = [t.contiguous() for t in (a[:, :132], w_gate_up[:, :132])]
    assert few(*odd, w_down) is None
    assert few(a, w_gate_up[:2 * 68].contiguous(), w_down[:, :68].contiguous()) is None
