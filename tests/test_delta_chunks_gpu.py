"""The delta rule by stretches of 64 tokens (long spans of a bfloat16 run) against the plain statement and the scan: spans around
whole stretches, states carried over steps, decays and erasures from none to all, keys that repeat, numbers that are not finite."""
import pytest
import torch

from plain.plain_kernels import PlainKernels
from test_chunk_scan_gpu import MIXED, STEPS, _Ctx, _mixed_ctx, _part

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
BF = torch.bfloat16


def _scan(kernels, chunks, *args):
    before, kernels.chunk_scans = kernels.chunk_scans, chunks
    try:
        return kernels.delta_rule_scan(*args)
    finally:
        kernels.chunk_scans = before


@pytest.mark.parametrize("H,w_shift,a_shift,same_keys", [(3, 0.0, 0.0, False), (1, -8.0, -8.0, False), (2, 8.0, 8.0, False), (2, -8.0, 8.0, True)])
def test_delta_rule(cuda_kernels, H, w_shift, a_shift, same_keys):
    D, HD, front = 64, 64 * H, 8
    g = torch.Generator().manual_seed(H)
    w0, ab, nw = torch.randn(HD, generator=g) + w_shift, torch.randn(HD, generator=g) + a_shift, 1 + 0.2 * torch.randn(HD, generator=g)
    states = [torch.zeros(4, front + HD * D, device=DEV) for _ in range(2)]
    state_p = torch.zeros(4, front + HD * D, dtype=F64)
    for lens, slots in STEPS:
        T = sum(lens)
        proj, w_raw = torch.randn(T, 5 * HD, generator=g), torch.randn(T, HD, generator=g)
        if same_keys:                                                           # every key nearly the one before: the system at its fullest
            proj[:, HD:2 * HD] = proj[:1, HD:2 * HD] + 0.05 * proj[:, HD:2 * HD]
        want = PlainKernels(wide=True).delta_rule_scan(proj.double(), w_raw.double(), w0, ab, nw, 1e-5, H, D, state_p[:, front:],
                                                       _Ctx(lens, slots, "cpu"), F64)
        for st, chunks in zip(states, (True, False)):
            before = cuda_kernels.launches
            y = _scan(cuda_kernels, chunks, proj.to(DEV), w_raw.to(DEV), w0.to(DEV), ab.to(DEV), nw.to(DEV), 1e-5, H, D, st[:, front:],
                      _Ctx(lens, slots, DEV), BF)
            assert cuda_kernels.launches - before == (4 if chunks else 3)
            assert float((y.double().cpu() - want).abs().max()) <= 2.0 ** -8 * max(1.0, float(want.abs().max()))
        # both make float32 sums of up to 300 terms: as near to the 64-bit ones as one another
        errors = [float((st.double().cpu() - state_p).norm() / state_p.norm()) for st in states]
        assert errors[0] <= 4 * errors[1] + 5e-7, errors
    assert float(states[0][1].abs().max()) == 0.0 and float(states[0][:, :front].abs().max()) == 0.0


@pytest.mark.parametrize("block", range(5))
def test_a_number_that_is_not_finite_reaches_what_follows_it(cuda_kernels, block):
    H, D, T, t0 = 2, 64, 200, 70
    HD = H * D
    g = torch.Generator().manual_seed(5)
    proj, w_raw = torch.randn(T, 5 * HD, generator=g), torch.randn(T, HD, generator=g)
    clean = proj.clone()
    proj[t0, block * HD + 3] = float("inf") if block < 3 else float("nan")       # r, k, v, g, a
    vec = [torch.randn(HD, generator=g).to(DEV) for _ in range(3)]
    results = []
    for rows, chunks in ((clean, True), (proj, True), (proj, False)):
        state = torch.zeros(1, HD * D, device=DEV)
        results.append((_scan(cuda_kernels, chunks, rows.to(DEV), w_raw.to(DEV), *vec, 1e-6, H, D, state, _Ctx((T,), (0,), DEV), BF), state))
    (y0, _), (y, state), (walk, state_w) = results
    assert torch.equal(y[:64], y0[:64]) and torch.equal(y[:, D:], y0[:, D:])      # stretches in front, the other head
    assert torch.equal(torch.isfinite(y), torch.isfinite(walk)) and torch.equal(torch.isfinite(state), torch.isfinite(state_w))
    fine = torch.isfinite(walk)
    assert bool(fine[:t0].all()) and not bool(fine.all())
    assert float((y.float() - walk.float())[fine].abs().max()) <= 2.0 ** -7 * float(walk.float()[fine].abs().max())


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_tiny_state_beside_one_that_is_not_finite(cuda_kernels, value):
    """Columns of a state do not meet.  Those beside an infinity are multiplied in float32, in which a sum of 64 terms around 2^-130
    is off by 64 halves of 2^-149 at most, in each of four stretches and their erased parts."""
    H, D, T = 2, 64, 200
    HD = H * D
    g = torch.Generator().manual_seed(9)
    proj, w_raw = torch.randn(T, 5 * HD, generator=g), torch.randn(T, HD, generator=g) - 6.0
    proj[:, 2 * HD:3 * HD] = 0.0
    vec = [torch.randn(HD, generator=g) for _ in range(3)]
    first = torch.randn(HD * D, generator=g) * 2.0 ** -130
    state, state_p = first[None].to(DEV).clone(), first[None].double()
    state[0, 5] = value                                                         # head 0, key channel 0, value channel 5
    PlainKernels(wide=True).delta_rule_scan(proj.double(), w_raw.double(), *vec, 1e-6, H, D, state_p, _Ctx((T,), (0,), "cpu"), F64)
    _scan(cuda_kernels, True, proj.to(DEV), w_raw.to(DEV), *(t.to(DEV) for t in vec), 1e-6, H, D, state, _Ctx((T,), (0,), DEV), BF)
    got, want = state.view(H, D, D).double().cpu(), state_p.view(H, D, D)
    assert not bool(got[0, :, 5].isfinite().any())
    beside = [0, 1, 2, 3, 4, 6, 7]
    assert float(want[0, :, beside].abs().max()) > 2.0 ** -136
    assert float((got - want)[0, :, beside].abs().max()) <= 4 * 2 * 64 * 2.0 ** -150


@pytest.mark.parametrize("tokens", [130, 640])
def test_no_less_exact_than_the_scan(cuda_kernels, tokens):
    """Parameters where trained models have them.  Both make float32 sums of the same numbers; a tenth for chance."""
    H, D = 4, 64
    HD = H * D
    g = torch.Generator().manual_seed(tokens)
    proj, w_raw = torch.randn(tokens, 5 * HD, generator=g), 0.5 * torch.randn(tokens, HD, generator=g)
    w0, ab, nw = torch.rand(HD, generator=g) * 7 - 6, 0.5 * torch.rand(HD, generator=g), torch.ones(HD)
    state_p = torch.zeros(1, HD * D, dtype=F64)
    PlainKernels(wide=True).delta_rule_scan(proj.double(), w_raw.double(), w0, ab, nw, 1e-6, H, D, state_p, _Ctx((tokens,), (0,), "cpu"), F64)
    errors = []
    for chunks in (True, False):
        state = torch.zeros(1, HD * D, device=DEV)
        _scan(cuda_kernels, chunks, *(t.to(DEV) for t in (proj, w_raw, w0, ab, nw)), 1e-6, H, D, state, _Ctx((tokens,), (0,), DEV), BF)
        errors.append(float((state.double().cpu() - state_p).norm() / state_p.norm()))
    assert errors[0] <= 1.1 * errors[1], errors


@pytest.mark.parametrize("block", [0, 1])
def test_products_that_a_scan_does_not_form(cuda_kernels, block):
    """Decays at their strongest, counted from a stretch's middle, take a query (a key) beyond float32 that a scan never scales."""
    H, D, T, t0 = 2, 64, 200, 64 if block == 0 else 127
    HD = H * D
    g = torch.Generator().manual_seed(7)
    proj, w_raw = torch.randn(T, 5 * HD, generator=g), torch.randn(T, HD, generator=g)
    proj[t0, block * HD:(block + 1) * HD] *= 1e33 if block == 0 else 1e18
    proj[t0, 2 * HD:3 * HD] *= 1.0 if block == 0 else 1e-18
    if block == 1:                                                              # k k^T beyond float32 only where the stretch multiplies
        proj[:, :HD] *= 1e18
    w0, ab, nw = torch.full((HD,), 8.0), torch.randn(HD, generator=g), torch.ones(HD)
    results = []
    for chunks in (True, False):
        state = torch.zeros(1, HD * D, device=DEV)
        y = _scan(cuda_kernels, chunks, *(t.to(DEV) for t in (proj, w_raw, w0, ab, nw)), 1e-6, H, D, state, _Ctx((T,), (0,), DEV), BF)
        results.append((y.double(), state.double()))
    (y, state), (walk, state_w) = results
    assert torch.equal(torch.isfinite(y), torch.isfinite(walk)) and bool(torch.isfinite(state_w).all())
    fine = torch.isfinite(walk)
    assert float((y - walk)[fine].abs().max()) <= 2.0 ** -7 * float(walk[fine].abs().max())
    assert float((state - state_w).abs().max()) <= 1e-5 * float(state_w.abs().max())


@pytest.mark.parametrize("beside", [False, True])
def test_long_spans_by_stretches_beside_short_ones(cuda_kernels, monkeypatch, beside):
    _part(cuda_kernels, monkeypatch, beside)
    H, D = 3, 64
    HD = H * D
    g = torch.Generator().manual_seed(8)
    vec = [torch.randn(HD, generator=g) for _ in range(3)]
    state, state_p = torch.zeros(4, HD * D, device=DEV), torch.zeros(4, HD * D, dtype=F64)
    for step, (lens, slots) in enumerate(MIXED):
        T = sum(lens)
        proj, w_raw = torch.randn(T, 5 * HD, generator=g), torch.randn(T, HD, generator=g)
        want = PlainKernels(wide=True).delta_rule_scan(proj.double(), w_raw.double(), *vec, 1e-5, H, D, state_p, _Ctx(lens, slots, "cpu"), F64)
        before = cuda_kernels.launches
        y = cuda_kernels.delta_rule_scan(proj.to(DEV), w_raw.to(DEV), *(t.to(DEV) for t in vec), 1e-5, H, D, state,
                                         _mixed_ctx(lens, slots, DEV), BF)
        assert cuda_kernels.launches - before == ((6, 6, 3) if beside else (4, 4, 3))[step]     # two more for the short spans; the scan alone
        # the norm divides by the size of a head's sums, which may be small
        assert float((y.double().cpu() - want).abs().max()) <= 2.0 ** -8 * max(1.0, float(want.abs().max()))
        assert float((state.double().cpu() - state_p).abs().max()) <= 5e-6 * max(1.0, float(state_p.abs().max()))


def test_one_product_is_rounded_once(cuda_kernels, monkeypatch):
    """Nothing decays and nothing is erased, one token's key and value alone: the state is their products, each off by its rounding (2^-24)
    and by what the small parts' sum cuts off (2^-28); six products of parts instead of eight leave out up to 2^-24.2."""
    H, D, T = 6, 64, 128
    HD = H * D
    g = torch.Generator().manual_seed(3)
    proj = torch.zeros(T, 5, H, D)
    proj[100, 1], proj[:, 2] = torch.randn(H, D, generator=g), torch.randn(T, H, D, generator=g)
    never = torch.full((HD,), -200.0, device=DEV)             # (sigmoid: 0)
    monkeypatch.setattr(cuda_kernels, "_delta_by_chunks", lambda *a: (1, 0))
    state = torch.zeros(1, HD * D, device=DEV)
    cuda_kernels.delta_rule_scan(proj.view(T, -1).to(DEV), torch.zeros(T, HD, device=DEV), never, never, torch.ones(HD, device=DEV), 1e-6, H, D,
                                 state, _Ctx((T,), (0,), DEV), BF)
    want = proj[100, 1].double()[:, :, None] * proj[100, 2].double()[:, None]    # [head, key channel, value channel]
    got = state.double().cpu().view(H, D, D)
    assert float(((got - want).abs() / want.abs()).max()) * 2.0 ** 24 <= 1.07
