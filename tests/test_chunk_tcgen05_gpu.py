"""Recurrences with a decay per head by stretches of 128 tokens on the tensor cores: what the stretches of 64 have to satisfy, and spans
around whole stretches, heads that share queries and keys, numbers that cannot be cut."""
import pytest
import torch

import test_chunk_scan_gpu as by_64
from plain.plain_kernels import PlainKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
SIZES = [("softplus_step", 4, 1, 128, 64), ("softplus_step", 2, 2, 64, 128), ("softplus_step", 2, 1, 128, 128), ("constant", 3, 3, 64, 128),
         ("constant", 2, 2, 128, 128), ("constant", 6, 2, 128, 64)]


@pytest.fixture(autouse=True)
def _always(cuda_kernels, monkeypatch):
    monkeypatch.setattr(cuda_kernels, "stretch", 128)


@pytest.mark.parametrize("mode,H,G,dk,dv", SIZES)
@pytest.mark.parametrize("spread", [1.0, 30.0])
def test_as_the_stretches_of_64(cuda_kernels, mode, H, G, dk, dv, spread):
    by_64.test_decay_scan(cuda_kernels, mode, H, G, dk, dv, spread)


@pytest.mark.parametrize("mode,H,G,dk,dv", SIZES)
def test_no_less_exact_than_the_scan(cuda_kernels, mode, H, G, dk, dv):
    by_64.test_no_less_exact_than_the_scan(cuda_kernels, mode, H, G, dk, dv)


@pytest.mark.parametrize("mode,H,G,dk,dv", SIZES)
def test_products_that_a_scan_does_not_form(cuda_kernels, mode, H, G, dk, dv):
    by_64.test_products_that_a_scan_does_not_form(cuda_kernels, mode, H, G, dk, dv)


@pytest.mark.parametrize("which,size", [("q", float("inf")), ("k", float("inf")), ("v", float("inf")), ("k", 3.4e38), ("v", 3.4e38)])
@pytest.mark.parametrize("mode,H,G,dk,dv", SIZES)
def test_a_number_that_cannot_be_cut(cuda_kernels, mode, H, G, dk, dv, which, size):
    """In the second of three stretches: nothing in front of it changes, what follows is what the scan gives.  (The largest numbers, whose
    upper part would round to infinity, meet small ones, so that no sum is beyond float32.)"""
    T, t0 = 300, 170
    g = torch.Generator().manual_seed(5)
    wide, raw = by_64._decay_inputs(mode, T, H, G, dk, dv, g, 1.0)
    if size < float("inf"):
        wide[t0, G * dk:] *= 1e-30
    wide[t0, {"q": 3, "k": G * dk + 3, "v": 2 * G * dk + 3}[which]] = size
    wide = wide.to(DEV)
    vec = [torch.rand(H, generator=g).to(DEV) for _ in range(3)]
    kw = {"rate": vec[0]} if mode == "constant" else {"step_bias": vec[0], "log_rate": vec[1], "skip": vec[2]}
    results = []
    for dtype in (torch.bfloat16, torch.float32):
        state = torch.zeros(1, H * dk * dv, device=DEV)
        out = cuda_kernels.decay_scan(wide[:, :G * dk], wide[:, G * dk:2 * G * dk], wide[:, 2 * G * dk:2 * G * dk + H * dv],
                                      None if raw is None else raw.to(DEV), state, by_64._Ctx((T,), (0,), DEV, dtype), heads=H, groups=G, dk=dk,
                                      dv=dv, decay=mode, **kw)
        results.append((out.double(), state.double()))
    (out, state), (walk, state_w) = results
    assert torch.equal(torch.isfinite(out), torch.isfinite(walk)) and torch.equal(torch.isfinite(state), torch.isfinite(state_w))
    fine = torch.isfinite(walk)
    assert bool(fine[:t0].all())
    size = torch.where(fine, walk.abs(), 0.0).amax(-1, keepdim=True)            # a row's: float32 sums of up to 300 terms
    assert float(((out - walk).abs() / size)[fine].max()) <= 1e-5


@pytest.mark.parametrize("mode,H,G,dk,dv", SIZES)
@pytest.mark.parametrize("lens", [(127,), (128,), (129,), (255, 1, 257), (64, 65, 63), (1, 1, 512)])
def test_spans_around_whole_stretches(cuda_kernels, monkeypatch, mode, H, G, dk, dv, lens):
    monkeypatch.setattr(cuda_kernels, "CHUNK_SCAN_MIN_SPAN", 1)
    g = torch.Generator().manual_seed(sum(lens) + H)
    slots = tuple(range(len(lens)))[::-1]
    vec = [torch.rand(H, generator=g) for _ in range(3)]
    kw = {"rate": 0.5 + 0.5 * vec[0]} if mode == "constant" else {"step_bias": vec[0] - 3, "log_rate": vec[1], "skip": vec[2]}
    on = {k: v.to(DEV) for k, v in kw.items()}
    wide, raw = by_64._decay_inputs(mode, sum(lens), H, G, dk, dv, g, 1.0)
    first = torch.randn(len(lens), H * dk * dv, generator=g)
    state, state_p = first.to(DEV), first.double()
    cut = lambda t: (t[:, :G * dk], t[:, G * dk:2 * G * dk], t[:, 2 * G * dk:2 * G * dk + H * dv])
    want = PlainKernels(wide=True).decay_scan(*cut(wide.double()), None if raw is None else raw.double(), state_p,
                                              by_64._Ctx(lens, slots, "cpu"), heads=H, groups=G, dk=dk, dv=dv, decay=mode, **kw).double()
    got = cuda_kernels.decay_scan(*cut(wide.to(DEV)), None if raw is None else raw.to(DEV), state, by_64._Ctx(lens, slots, DEV), heads=H, groups=G,
                                  dk=dk, dv=dv, decay=mode, **on)
    for a, b in ((got, want), (state, state_p)):             # float32 sums of up to 512 terms
        assert float((a.double().cpu() - b).abs().max()) <= 5e-6 * max(1.0, float(b.abs().max()))


def test_which_steps_take_them(cuda_kernels):
    rule = cuda_kernels.lib.ifx_chunk_scan_takes_128
    assert not rule(300, 1, 1, 12, 128) and rule(512, 1, 1, 12, 128) and rule(128, 1, 1, 28, 128)
    assert not rule(300, 32, 128, 12, 64)


def _off_by(got, want):
    """The largest relative error in units of 2^-24 (one rounding is at most one of them)."""
    at = want != 0
    return float(((got.double() - want).abs()[at] / want.abs()[at]).max()) * 2.0 ** 24


@pytest.mark.parametrize("H,G,dk,dv", [(2, 2, 64, 128), (2, 2, 128, 128), (6, 2, 128, 64)])
def test_one_product_is_rounded_once(cuda_kernels, H, G, dk, dv):
    """Without decay, one token's key and value alone: the state is their products, and one channel of a query alone reads products of the
    state.  Whatever parts operands are cut into, a product of two numbers is off by its rounding (2^-24) and by what is left out of and
    cut off the small parts (eight ends of sums of 2^-8, 2^-28; six products of parts instead of eight leave out up to 2^-24.2)."""
    T = 300
    g = torch.Generator().manual_seed(dk + dv)
    q, k, v = torch.zeros(T, G, dk), torch.zeros(T, G, dk), torch.zeros(T, H, dv)
    k[290], v[290] = torch.randn(G, dk, generator=g), torch.randn(H, dv, generator=g)
    rate = torch.ones(H, device=DEV)
    kw = dict(heads=H, groups=G, dk=dk, dv=dv, decay="constant", rate=rate)
    state = torch.zeros(1, H * dk * dv, device=DEV)
    cuda_kernels.decay_scan(q.view(T, -1).to(DEV), k.view(T, -1).to(DEV), v.view(T, -1).to(DEV), None, state, by_64._Ctx((T,), (0,), DEV), **kw)
    keys = k[290].repeat_interleave(H // G, 0).double()
    want = v[290].double()[:, :, None] * keys[:, None]                           # [head, value channel, key channel]
    assert _off_by(state.cpu().view(H, dv, dk), want) <= 1.07
    q = torch.zeros(T, G, dk)
    which = torch.randint(0, dk, (T, G, 1), generator=g)
    q.scatter_(2, which, torch.randn(T, G, 1, generator=g))
    held = torch.randn(H, dv, dk, generator=g)
    out = cuda_kernels.decay_scan(q.view(T, -1).to(DEV), torch.zeros(T, G * dk, device=DEV), v.view(T, -1).to(DEV), None,
                                  held.reshape(1, -1).to(DEV), by_64._Ctx((T,), (0,), DEV), **kw)
    want = torch.einsum("thk,hvk->thv", q.double().repeat_interleave(H // G, 1), held.double())
    assert _off_by(out.cpu().view(T, H, dv)[:128], want[:128]) <= 1.07          # (the first stretch: the state as it was)
