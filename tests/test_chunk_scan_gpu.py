"""The recurrences by stretches of 64 tokens (long spans of a bfloat16 run) against the plain statement and the token-by-token
kernels: spans around whole stretches, states carried over steps, decays from none to one, numbers that are not finite."""
import pytest
import torch

from plain.plain_kernels import PlainKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


class _Ctx:
    """What the scans read of a step context of a bfloat16 run."""

    def __init__(self, lens, slots, device, dtype=torch.bfloat16):
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        self.cu_seqlens = torch.tensor(cu, dtype=torch.int32, device=device)
        self.req_slot = torch.tensor(slots, dtype=torch.int32, device=device)
        self.num_requests, self.max_span, self.dtype = len(lens), max(lens), dtype


STEPS = [((128, 1, 65), (3, 0, 2)), ((1, 300), (3, 2)), ((191, 129, 64), (2, 3, 0))]


def _decay_inputs(mode, T, H, G, dk, dv, g, spread):
    wide = torch.randn(T, 2 * G * dk + H * dv + 4, generator=g)                 # q | k | v as slices of wider rows
    raw = None if mode == "constant" else spread * torch.randn(T, H * dk if mode == "sigmoid_root" else H, generator=g)
    return wide, raw


@pytest.mark.parametrize("spread", [1.0, 30.0])
@pytest.mark.parametrize("mode,H,G,dk,dv", [("sigmoid_root", 2, 2, 64, 128), ("sigmoid_root", 1, 1, 128, 64), ("softplus_step", 4, 1, 128, 64),
                                            ("softplus_step", 2, 2, 64, 64), ("constant", 3, 3, 64, 128), ("constant", 2, 2, 128, 128)])
def test_decay_scan(cuda_kernels, mode, H, G, dk, dv, spread):
    """`spread` 30: decays that are zero or one within a few tokens."""
    g = torch.Generator().manual_seed(H * 1000 + dk + dv)
    bias, rate, skip = torch.randn(H, generator=g), torch.rand(H, generator=g) * 2 - 1, torch.randn(H, generator=g)
    const = torch.cat([torch.rand(H, generator=g)[1:] * 0.5 + 0.5, torch.ones(1)])
    kw = {"sigmoid_root": {"tau": 3.0, "q_scale": dk ** -0.5}, "softplus_step": {"step_bias": bias, "log_rate": rate, "skip": skip},
          "constant": {"rate": const}}[mode]
    on = {k: v.to(DEV) if torch.is_tensor(v) else v for k, v in kw.items()}
    front = 8                                                                   # floats of another part's state first
    states = [torch.zeros(4, front + H * dk * dv, device=DEV) for _ in range(2)]
    state_p = torch.zeros(4, front + H * dk * dv, dtype=F64)
    for lens, slots in STEPS:
        wide, raw = _decay_inputs(mode, sum(lens), H, G, dk, dv, g, spread)
        cut = lambda t: (t[:, :G * dk], t[:, G * dk:2 * G * dk], t[:, 2 * G * dk:2 * G * dk + H * dv])
        want = PlainKernels(wide=True).decay_scan(*cut(wide.double()), None if raw is None else raw.double(), state_p[:, front:],
                                                  _Ctx(lens, slots, "cpu"), heads=H, groups=G, dk=dk, dv=dv, decay=mode, **kw).double()
        before = cuda_kernels.launches
        got, walk = (cuda_kernels.decay_scan(*cut(wide.to(DEV)), None if raw is None else raw.to(DEV), st[:, front:],
                                             _Ctx(lens, slots, DEV, dtype), heads=H, groups=G, dk=dk, dv=dv, decay=mode, **on)
                     for st, dtype in zip(states, (torch.bfloat16, torch.float32)))
        # both make float32 sums of up to 300 terms: as near to the 64-bit ones as one another
        scale, size = max(1.0, float(want.abs().max())), max(1.0, float(state_p.abs().max()))
        errors = [float((t.double().cpu() - want).abs().max()) / scale for t in (got, walk)]
        assert errors[0] <= 2 * errors[1] + 1e-6, errors
        errors = [float((t.double().cpu() - state_p).abs().max()) / size for t in states]
        assert errors[0] <= 2 * errors[1] + 1e-6, errors
        assert cuda_kernels.launches > before
    assert float(states[0][1].abs().max()) == 0.0 and float(states[0][:, :front].abs().max()) == 0.0


@pytest.mark.parametrize("shift", [-1.0, 3.0, -6.0])
@pytest.mark.parametrize("H,D", [(3, 64), (1, 128)])
def test_wkv_scan(cuda_kernels, H, D, shift):
    """`shift` 3: decays near zero; -6: near one."""
    HD, C = H * D, 40
    g = torch.Generator().manual_seed(H + D)
    w0, u, nw = torch.randn(HD, generator=g) + shift, 0.5 * torch.randn(HD, generator=g), 1 + 0.2 * torch.randn(HD, generator=g)
    states = [torch.zeros(4, HD * D + C, device=DEV) for _ in range(2)]
    state_p = torch.zeros(4, HD * D + C, dtype=F64)
    for lens, slots in STEPS:
        T = sum(lens)
        wide, w_raw, x = torch.randn(T, 4 * HD, generator=g), torch.randn(T, HD, generator=g), torch.randn(T, C, generator=g)
        cut = lambda t: tuple(t[:, i * HD:(i + 1) * HD] for i in range(4))
        r, k, v, gate = cut(wide)
        want = PlainKernels(wide=True).wkv_scan(r, k, v, w_raw, gate, w0, u, nw, 1e-5, H, D, state_p, HD * D, x.double(),
                                                _Ctx(lens, slots, "cpu"), F64)
        on = wide.to(DEV)
        for st, chunks in zip(states, (True, False)):
            cuda_kernels.chunk_scans = chunks
            try:
                y = cuda_kernels.wkv_scan(*cut(on)[:3], w_raw.to(DEV), cut(on)[3], w0.to(DEV), u.to(DEV), nw.to(DEV), 1e-5, H, D, st,
                                          HD * D, x.to(DEV), _Ctx(lens, slots, DEV), torch.bfloat16)
            finally:
                cuda_kernels.chunk_scans = True
            assert float((y.double().cpu() - want).abs().max()) <= 2.0 ** -8 * max(1.0, float(want.abs().max()))
        errors = [float((st.double().cpu() - state_p).abs().max()) / max(1.0, float(state_p.abs().max())) for st in states]
        assert errors[0] <= 2 * errors[1] + 1e-6, errors
    assert float(states[0][1].abs().max()) == 0.0


@pytest.mark.parametrize("which", ["q", "k", "v"])
@pytest.mark.parametrize("mode,H,G,dk,dv", [("sigmoid_root", 2, 2, 64, 64), ("softplus_step", 2, 1, 128, 64)])
def test_a_number_that_is_not_finite_reaches_what_follows_it(cuda_kernels, mode, H, G, dk, dv, which):
    """As in the scan token by token: nothing in front of it, and the same tokens and channels behind it."""
    T, t0 = 200, 70
    g = torch.Generator().manual_seed(5)
    wide, raw = _decay_inputs(mode, T, H, G, dk, dv, g, 1.0)
    wide[t0, {"q": 3, "k": G * dk + 3, "v": 2 * G * dk + 3}[which]] = float("inf")
    wide = wide.to(DEV)
    vec = [torch.rand(H, generator=g).to(DEV) for _ in range(3)]
    kw = {"tau": 3.0} if mode == "sigmoid_root" else {"step_bias": vec[0], "log_rate": vec[1], "skip": vec[2]}
    results = []
    for dtype in (torch.bfloat16, torch.float32):
        state = torch.zeros(1, H * dk * dv, device=DEV)
        out = cuda_kernels.decay_scan(wide[:, :G * dk], wide[:, G * dk:2 * G * dk], wide[:, 2 * G * dk:2 * G * dk + H * dv], raw.to(DEV),
                                      state, _Ctx((T,), (0,), DEV, dtype), heads=H, groups=G, dk=dk, dv=dv, decay=mode, **kw)
        results.append((out, state))
    (out, state), (walk, state_w) = results
    assert torch.equal(torch.isfinite(out), torch.isfinite(walk)) and torch.equal(torch.isfinite(state), torch.isfinite(state_w))
    fine = torch.isfinite(walk)
    assert bool(fine[:t0].all()) and not bool(fine.all())
    assert float((out - walk)[fine].abs().max()) <= 1e-5 * float(walk[fine].abs().max())


def test_which_spans_go_by_stretches(cuda_kernels):
    """Short spans, a float32 run, other sizes and rows off a 16-byte boundary keep the token-by-token kernels."""
    row = torch.zeros(4, 65, device=DEV)
    fits = lambda ctx, dtype, dk=64, dv=64, rows=row[:, :64].contiguous(): cuda_kernels._scans_by_chunks(dtype, ctx, 2, dk, dv, rows)
    long, short = _Ctx((500, 2), (0, 1), DEV), _Ctx((cuda_kernels.CHUNK_SCAN_MIN_SPAN - 1,), (0,), DEV)
    assert fits(long, torch.bfloat16) and fits(long, torch.bfloat16, 128, 192)
    assert not fits(long, torch.float32) and not fits(short, torch.bfloat16)
    assert not fits(long, torch.bfloat16, 96) and not fits(long, torch.bfloat16, 64, 96)
    assert not fits(long, torch.bfloat16, rows=row[:, 1:]) and not fits(long, torch.bfloat16, rows=row[:, :64])


@pytest.mark.parametrize("mode,H,G,dk,dv", [("sigmoid_root", 2, 2, 64, 128), ("softplus_step", 4, 1, 128, 64), ("constant", 3, 3, 128, 128),
                                            ("constant", 3, 3, 64, 128)])
def test_no_less_exact_than_the_scan(cuda_kernels, mode, H, G, dk, dv):
    """Parameters where trained models have them.  Both make float32 sums of the same numbers; a tenth for chance."""
    T = 500
    g = torch.Generator().manual_seed(dk + dv)
    uniform = lambda lo, hi, *s: torch.rand(*s, generator=g) * (hi - lo) + lo
    wide, raw = _decay_inputs(mode, T, H, G, dk, dv, g, 0.5)
    if mode == "sigmoid_root":
        raw += uniform(-2.0, 4.0, H * dk)
    kw = {"sigmoid_root": {"tau": 16.0, "q_scale": dk ** -0.5}, "constant": {"rate": torch.tensor([1 - 2 ** (-5 - 5 * i / H) for i in range(H)])},
          "softplus_step": {"step_bias": uniform(-6, -2, H), "log_rate": uniform(0, 2.7, H), "skip": uniform(0, 0.2, H)}}[mode]
    on = {k: v.to(DEV) if torch.is_tensor(v) else v for k, v in kw.items()}
    cut = lambda t: (t[:, :G * dk], t[:, G * dk:2 * G * dk], t[:, 2 * G * dk:2 * G * dk + H * dv])
    state_p = torch.zeros(1, H * dk * dv, dtype=F64)
    want = PlainKernels(wide=True).decay_scan(*cut(wide.double()), None if raw is None else raw.double(), state_p, _Ctx((T,), (0,), "cpu"),
                                              heads=H, groups=G, dk=dk, dv=dv, decay=mode, **kw).double()
    errors = []
    for dtype in (torch.bfloat16, torch.float32):
        state = torch.zeros(1, H * dk * dv, device=DEV)
        out = cuda_kernels.decay_scan(*cut(wide.to(DEV)), None if raw is None else raw.to(DEV), state, _Ctx((T,), (0,), DEV, dtype), heads=H,
                                      groups=G, dk=dk, dv=dv, decay=mode, **on)
        errors.append([float((a.double().cpu() - b).norm() / b.norm()) for a, b in ((out, want), (state, state_p))])
    assert errors[0][0] <= 1.1 * errors[1][0] and errors[0][1] <= 1.1 * errors[1][1], errors


@pytest.mark.parametrize("mode,H,G,dk,dv", [("sigmoid_root", 2, 2, 64, 64), ("softplus_step", 2, 1, 128, 64), ("constant", 2, 2, 64, 64)])
def test_products_that_a_scan_does_not_form(cuda_kernels, mode, H, G, dk, dv):
    """A query and a key whose product is beyond float32, beside a value that brings the state back into range: finite in the scan."""
    T, t0 = 200, 70
    g = torch.Generator().manual_seed(6)
    wide, raw = _decay_inputs(mode, T, H, G, dk, dv, g, 1.0)
    wide[t0, :2 * G * dk] *= 1e25
    wide[t0, 2 * G * dk:] *= 1e-30
    wide = wide.to(DEV)
    vec = [torch.rand(H, generator=g).to(DEV) for _ in range(3)]
    kw = {"sigmoid_root": {"tau": 3.0}, "softplus_step": {"step_bias": vec[0], "log_rate": vec[1], "skip": vec[2]},
          "constant": {"rate": vec[0]}}[mode]
    results = []
    for dtype in (torch.bfloat16, torch.float32):
        state = torch.zeros(1, H * dk * dv, device=DEV)
        out = cuda_kernels.decay_scan(wide[:, :G * dk], wide[:, G * dk:2 * G * dk], wide[:, 2 * G * dk:2 * G * dk + H * dv],
                                      None if raw is None else raw.to(DEV), state, _Ctx((T,), (0,), DEV, dtype), heads=H, groups=G, dk=dk,
                                      dv=dv, decay=mode, **kw)
        results.append((out.double(), state.double()))
    (out, state), (walk, state_w) = results
    assert bool(torch.isfinite(walk).all()) and bool(torch.isfinite(out).all())
    size = walk.abs().amax(-1, keepdim=True)                                    # float32 sums of up to 200 terms
    assert float(((out - walk).abs() / size).max()) <= 1e-4
    assert float((state - state_w).abs().max()) <= 1e-5 * float(state_w.abs().max())


MIXED = [((300, 1, 130, 90), (3, 0, 2, 1)), ((1, 300, 1, 5), (3, 2, 0, 1)), ((1, 1, 1, 1), (0, 1, 2, 3))]


def _mixed_ctx(lens, slots, device):
    ctx = _Ctx(lens, slots, device)
    ctx.spans = [(0, n) for n in lens]
    return ctx


def _part(cuda_kernels, monkeypatch, beside):
    """All spans of a step by stretches, or the long ones beside the scan for the others."""
    plan = lambda short: (128, short) if beside and short else (1, 0)
    monkeypatch.setattr(cuda_kernels, "stretches_pay", lambda longest, blocks, cheap, short, *more: plan(short))
    monkeypatch.setattr(cuda_kernels, "delta_stretches_pay", lambda heads, tokens, requests, longest, short, *more: plan(short))


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("mode,H,G,dk,dv", [("sigmoid_root", 2, 2, 64, 128), ("softplus_step", 2, 1, 128, 64), ("constant", 3, 3, 64, 64)])
def test_long_spans_by_stretches_beside_short_ones(cuda_kernels, monkeypatch, mode, H, G, dk, dv, beside):
    _part(cuda_kernels, monkeypatch, beside)
    g = torch.Generator().manual_seed(dk)
    vec = [torch.rand(H, generator=g) for _ in range(3)]
    kw = {"sigmoid_root": {"tau": 3.0}, "softplus_step": {"step_bias": vec[0], "log_rate": vec[1], "skip": vec[2]},
          "constant": {"rate": vec[0]}}[mode]
    on = {k: v.to(DEV) if torch.is_tensor(v) else v for k, v in kw.items()}
    state, state_p = torch.zeros(4, H * dk * dv, device=DEV), torch.zeros(4, H * dk * dv, dtype=F64)
    for step, (lens, slots) in enumerate(MIXED):
        wide, raw = _decay_inputs(mode, sum(lens), H, G, dk, dv, g, 1.0)
        cut = lambda t: (t[:, :G * dk], t[:, G * dk:2 * G * dk], t[:, 2 * G * dk:2 * G * dk + H * dv])
        want = PlainKernels(wide=True).decay_scan(*cut(wide.double()), None if raw is None else raw.double(), state_p, _Ctx(lens, slots, "cpu"),
                                                  heads=H, groups=G, dk=dk, dv=dv, decay=mode, **kw).double()
        before = cuda_kernels.launches
        got = cuda_kernels.decay_scan(*cut(wide.to(DEV)), None if raw is None else raw.to(DEV), state, _mixed_ctx(lens, slots, DEV), heads=H,
                                      groups=G, dk=dk, dv=dv, decay=mode, **on)
        # three for the stretches, the scan, and its decays ahead of it where its longest span has 64 tokens and they are not constant
        assert cuda_kernels.launches - before == (((5 if mode != "constant" else 4), 4, 1) if beside else (3, 3, 1))[step]
        for a, b in ((got, want), (state, state_p)):                            # float32 sums of up to 300 terms
            assert float((a.double().cpu() - b).abs().max()) <= 5e-6 * max(1.0, float(b.abs().max()))


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("H,D", [(3, 64), (1, 128)])
def test_wkv_of_long_and_short_spans(cuda_kernels, monkeypatch, H, D, beside):
    _part(cuda_kernels, monkeypatch, beside)
    HD, C = H * D, 40
    g = torch.Generator().manual_seed(H)
    w0, u, nw = torch.randn(HD, generator=g), 0.5 * torch.randn(HD, generator=g), 1 + 0.2 * torch.randn(HD, generator=g)
    state, state_p = torch.zeros(4, HD * D + C, device=DEV), torch.zeros(4, HD * D + C, dtype=F64)
    for step, (lens, slots) in enumerate(MIXED):
        T = sum(lens)
        r, k, v, gate, w_raw = (torch.randn(T, HD, generator=g) for _ in range(5))
        x = torch.randn(T, C, generator=g)
        want = PlainKernels(wide=True).wkv_scan(r, k, v, w_raw, gate, w0, u, nw, 1e-5, H, D, state_p, HD * D, x.double(),
                                                _Ctx(lens, slots, "cpu"), F64)
        before = cuda_kernels.launches
        y = cuda_kernels.wkv_scan(*(t.to(DEV) for t in (r, k, v, w_raw, gate, w0, u, nw)), 1e-5, H, D, state, HD * D, x.to(DEV),
                                  _mixed_ctx(lens, slots, DEV), torch.bfloat16)
        assert cuda_kernels.launches - before == ((5, 5, 1) if beside else (4, 4, 1))[step]
        assert float((y.double().cpu() - want).abs().max()) <= 2.0 ** -8 * max(1.0, float(want.abs().max()))
        assert float((state.double().cpu() - state_p).abs().max()) <= 5e-6 * max(1.0, float(state_p.abs().max()))


def test_rows_off_a_16_byte_boundary_go_by_the_scan(cuda_kernels):
    """The kernels of long spans refuse them before they touch anything; nothing is done twice."""
    T, H, d = 200, 2, 64
    g = torch.Generator().manual_seed(9)
    rows, rate = torch.randn(T, 3 * H * d + 1, generator=g).to(DEV), torch.full((H,), 0.9, device=DEV)
    results = []
    for dtype in (torch.bfloat16, torch.float32):
        state = torch.ones(1, H * d * d, device=DEV)
        cut = [rows[:, 1 + i * H * d:1 + (i + 1) * H * d] for i in range(3)]
        results.append((cuda_kernels.decay_scan(*cut, None, state, _Ctx((T,), (0,), DEV, dtype), heads=H, groups=H, dk=d, dv=d,
                                                decay="constant", rate=rate), state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
