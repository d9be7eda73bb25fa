"""The float32 product on the tensor cores (operands in three bfloat16 parts) at its edges: rows around its tiles of tokens and
the blocks of rows worked on at a time, columns and K that fill no tile, K whole and in slices."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def operands(M, N, K, seed=0):
    g = torch.Generator().manual_seed(M * 7 + N + K + seed)
    return tuple(torch.randn(n, generator=g).to(DEV) for n in ((M, K), (N, K), (N,)))


def bound(a, w):
    """Products left out: three below 2^-24 of one each.  A chunk of 64 k: 4 additions of its largest products into its accumulator that
    may cut off up to 2^-22 each (aligned products, then the sum), 320 of the others, 2^-7 of them, into theirs.  The chunks' and
    slices' rounded additions: 2^-24 each."""
    K = a.shape[1]
    return (3 * 2.0 ** -24 + (4 + 320 * 2.0 ** -7) * 2.0 ** -22 + (K / 64 + 150) * 2.0 ** -24) * (a.double().abs() @ w.double().abs().t()) + 1e-30


# 1,700 columns: slices of K; 19,000: 149 tiles of columns, K whole
@pytest.mark.parametrize("M,N,K", [(1, 1700, 1288), (16, 1700, 1280), (17, 1699, 1344), (33, 1700, 4104), (64, 19000, 1280),
                                   (65, 18951, 1288), (127, 1700, 1288), (129, 1700, 1288), (333, 19000, 1288), (1030, 1700, 1288),
                                   (2, 70, 30008)])
def test_against_64_bits(cuda_kernels, M, N, K):
    assert cuda_kernels.float32_by_parts(N, K)
    a, w, bias = operands(M, N, K)
    want, chain = a.double() @ w.double().t(), cuda_kernels.linear_generic(a, w)
    for b in (None, bias):
        got = cuda_kernels.linear(a, w, b).double()
        exact = want if b is None else want + b.double()
        assert bool(((got - exact).abs() <= bound(a, w) + 2.0 ** -24 * exact.abs()).all())
    assert float((cuda_kernels.linear(a, w).double() - want).norm()) <= float((chain.double() - want).norm())
    cuda_kernels.check_errors()


@pytest.mark.parametrize("N,K", [(1700, 1288), (19000, 1280)])
def test_rows_do_not_depend_on_their_number(cuda_kernels, N, K):
    a, w, bias = operands(1100, N, K)
    whole = cuda_kernels.linear(a, w, bias)
    for n in (1, 16, 40, 97, 200, 1024):
        assert torch.equal(cuda_kernels.linear(a[:n].contiguous(), w, bias), whole[:n])


@pytest.mark.parametrize("N", [1700, 19000])
def test_not_finite_tiny_and_huge(cuda_kernels, N):
    """Rows whose parts leave bfloat16's range, or are no numbers, come out as from the chain of multiply-adds; the others as ever."""
    a, w, _ = operands(40, N, 1288, seed=1)
    clean = cuda_kernels.linear(a, w)
    a[3, 7], a[4, 1287], a[5, 0] = float("inf"), float("nan"), -float("inf")
    w[11, 3] = float("inf")
    a[6] *= 2.0 ** -118
    a[7] *= 2.0 ** 122                                        # sums beyond the largest float32 in some columns
    a[8] = 0.0
    a[9, :], a[9, 2] = 0.0, 3.4e38
    got, chain = cuda_kernels.linear(a, w), cuda_kernels.linear_generic(a, w)
    for r in (3, 4, 5, 6, 8):
        assert torch.equal(got[r].nan_to_num(nan=7.0), chain[r].nan_to_num(nan=7.0)) and torch.equal(got[r].isnan(), chain[r].isnan())
    # a sum that goes beyond the largest float32 and comes back within a chunk may be finite here alone: then it is the right one
    want, most = a.double() @ w.double().t(), bound(a, w)
    for r in (7, 9):
        f = got[r].isfinite()
        assert bool(f[chain[r].isfinite()].all()) and torch.equal(got[r][~f].nan_to_num(nan=7.0), chain[r][~f].nan_to_num(nan=7.0))
        assert bool(f.any()) and bool(((got[r].double() - want[r]).abs() <= most[r])[f].all())
    keep = torch.ones(40, dtype=torch.bool, device=DEV)
    keep[3:10] = False
    cols = torch.arange(N, device=DEV) != 11
    assert torch.equal(got[keep][:, cols], clean[keep][:, cols])
    assert not bool(got[keep][:, 11].isfinite().any())


@pytest.mark.parametrize("N,K", [(1700, 1288), (19000, 1280), (1536, 8960)])
@pytest.mark.parametrize("terms", [1, 2, 4, 8])
def test_rows_of_few_terms_round_as_the_chain(cuda_kernels, N, K, terms):
    """Errors that do not average out.  One term: what is left out (2^-24) and one rounding, the smaller products' cut off below; more:
    a rounding or two beyond the chain's (2-norm up to 1.5 of its, 2 to 4 where parts are cut off instead of rounded)."""
    a, w, _ = operands(40, N, K, seed=terms)
    g = torch.Generator().manual_seed(terms)
    keep = torch.zeros(40, K).scatter_(1, torch.rand(40, K, generator=g).argsort(1)[:, :terms], 1.0).to(DEV)
    a *= keep
    a[0], w[:8] = keep[0] * (1 + 2.0 ** -7 - 2.0 ** -23), 1 + 2.0 ** -7 - 2.0 ** -23      # what mantissas of this kind leave out adds up
    want = a.double() @ w.double().t()
    got, chain = cuda_kernels.linear(a, w).double() - want, cuda_kernels.linear_generic(a, w).double() - want
    assert float(got.norm()) <= 1.5 * float(chain.norm())
    if terms == 1:
        assert bool((got.abs() <= (2 * 2.0 ** -24 + 20 * 2.0 ** -30) * want.abs()).all())


@pytest.mark.parametrize("N", [1700, 19000])
@pytest.mark.parametrize("small,large", [(-118, 100), (-125, 110), (-128, 60), (-140, 120), (-146, 20), (-133, 0), (-100, 4), (-70, -60)])
def test_tiny_numbers_against_large_ones(cuda_kernels, N, small, large):
    """Their lower parts are below bfloat16's range, whatever the result is."""
    a, w, bias = operands(33, N, 1288, seed=2)
    for x, y in ((a * 2.0 ** small, w * 2.0 ** large), (a * 2.0 ** large, w * 2.0 ** small)):
        for b in (None, bias):
            got, chain = cuda_kernels.linear(x, y, b), cuda_kernels.linear_generic(x, y, b)
            assert bool(chain.isfinite().all()) and bool((chain != 0).any()) and torch.equal(got, chain)
    # among numbers of ordinary size they are next to nothing, and stay that
    x, y = a.clone(), w * 2.0 ** min(large, 28)
    x[:, ::3] *= 2.0 ** small
    assert bool(((cuda_kernels.linear(x, y).double() - x.double() @ y.double().t()).abs() <= bound(x, y)).all())
    cuda_kernels.check_errors()


@pytest.mark.parametrize("N", [1700, 19000])
def test_rows_of_zeros(cuda_kernels, N):
    a, w, bias = operands(100, N, 1288, seed=3)
    a[5:50], w[7], w[9], w[N - 1] = 0.0, 0.0, -0.0, 0.0
    a[60, 3], w[30, 5], a[99, :], a[99, 1287] = float("inf"), float("nan"), 0.0, 2.0 ** -140
    got, chain = cuda_kernels.linear(a, w, bias), cuda_kernels.linear_generic(a, w, bias)
    for x, y in ((got[5:50], chain[5:50]), (got[:, [7, 9, 30, N - 1]], chain[:, [7, 9, 30, N - 1]]), (got[60], chain[60]), (got[99], chain[99])):
        assert torch.equal(x.nan_to_num(nan=7.0), y.nan_to_num(nan=7.0)) and torch.equal(x.isnan(), y.isnan())


@pytest.mark.parametrize("N,K,rows", [(1536, 8960, 512), (3584, 18944, 256), (1700, 1288, 1024), (256, 16384, 384), (40, 262144, 32)])
def test_scratch_is_bounded(cuda_kernels, N, K, rows):
    """64 MB: more rows go in portions, whose results are the same bits."""
    assert cuda_kernels.float32_by_parts(N, K)
    a, w, bias = operands(rows + 5, N, K)
    room = cuda_kernels.lib.ifx_gemm_f32_split_scratch
    assert room(rows + 5, N, K) == room(rows, N, K) > room(rows - 1, N, K) and room(5000, N, K) <= 64 << 20
    whole = cuda_kernels.linear(a, w, bias)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = cuda_kernels.linear(a, w, bias)
    assert torch.cuda.max_memory_allocated() - before - out.numel() * 4 <= room(rows, N, K) + 4096
    assert torch.equal(out, whole) and torch.equal(cuda_kernels.linear(a[rows - 3:].contiguous(), w, bias), whole[rows - 3:])
    cuda_kernels.check_errors()


@pytest.mark.parametrize("M,N,K", [(33, 19000, 2048), (40, 18950, 2112), (17, 1536, 12288), (5, 1536, 12352)])
def test_whole_groups_of_chunks(cuda_kernels, M, N, K):
    """The smaller products' accumulator is added every 16 chunks of 64: 32 and 33 chunks, slices of 16 and of 17."""
    a, w, bias = operands(M, N, K)
    want = a.double() @ w.double().t() + bias.double()
    assert bool(((cuda_kernels.linear(a, w, bias).double() - want).abs() <= bound(a, w) + 2.0 ** -24 * want.abs()).all())
    cuda_kernels.check_errors()
