"""Kernels that go over rows by 16 bytes at a time, at the sizes where their ways part: norm and gate behind a recurrence, activated
columns, mixes of neighbouring rows, normed and turned latents; each against the statement in 64 bits."""
import pytest
import torch

from plain.plain_kernels import PlainKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
# a result of 32-bit sums of up to 10,000 terms and a few roundings more; the same stored in bfloat16
TOL = {torch.float32: 4e-6, torch.bfloat16: 2.0 ** -8}


def _close(got, want, dtype):
    scale = max(1.0, float(want.abs().max()))
    err = float(((got.double().cpu() - want).abs() / want.abs().clamp(min=0.05 * scale)).max())
    assert err <= TOL[dtype], err


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,groups,part", [(1, 24, 64), (803, 25, 64), (2400, 7, 64), (5, 3, 128), (1601, 12, 128), (9, 5, 96), (3, 2, 256), (4, 2, 260),
                                           (3, 1, 258), (7, 1, 1536), (2, 3, 8192), (2, 1, 8196)])
@pytest.mark.parametrize("gate_first,kind,off", [(False, "sigmoid", 0), (True, "silu", 4), (False, "silu", 1)])
def test_norm_and_gate(cuda_kernels, dtype, T, groups, part, gate_first, kind, off):
    """`off`: the gates' first column in their wider rows (1: not on a 16-byte boundary)."""
    g = torch.Generator().manual_seed(T * 31 + part)
    C = groups * part
    y, wide = torch.randn(T, C, generator=g), 3 * torch.randn(T, C + 8, generator=g)
    w = 1 + 0.3 * torch.randn(C if off else part, generator=g)
    gate = wide[:, off:off + C].double()
    gate = torch.sigmoid(gate) * (gate if kind == "silu" else 1.0)
    v = y.double() * (gate if gate_first else 1.0)
    v = v.view(T, groups, part)
    v = (v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-5) * w.double().view(-1, part)).reshape(T, C)
    got = cuda_kernels.gated_groupnorm(y.to(DEV), wide.to(DEV)[:, off:off + C], w.to(DEV), 1e-5, groups=groups, gate_first=gate_first,
                                       out_dtype=dtype, kind=kind)
    _close(got, v if gate_first else v * gate, dtype)


@pytest.mark.parametrize("T,width,acted", [(128, 4, 4), (127, 6144, 4608), (130, 6144, 4608), (200, 2052, 2048), (131, 2048, 2048), (129, 4100, 0),
                                           (140, 515, 512)])
def test_activated_columns(cuda_kernels, T, width, acted):
    rows = 4 * torch.randn(T, width, generator=torch.Generator().manual_seed(width))
    rows[0, 0], rows[1, 1] = -200.0, 200.0
    want = rows.double()
    want[:, :acted] *= torch.sigmoid(want[:, :acted])
    on = rows.to(DEV)
    got = cuda_kernels.silu_columns(on, acted, None)
    assert got.data_ptr() == on.data_ptr()
    _close(got, want, torch.float32)


class _Ctx:
    def __init__(self, spans, slots, device):
        lens = [n for _, n in spans]
        self.cu_seqlens = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=device)
        self.token_req = torch.tensor([r for r, n in enumerate(lens) for _ in range(n)], dtype=torch.int32, device=device)
        self.req_slot = torch.tensor(slots, dtype=torch.int32, device=device)
        self.positions = torch.tensor([s + i for s, n in spans for i in range(n)], dtype=torch.int32, device=device)
        self.num_requests, self.max_span, self.spans = len(lens), max(lens), spans
        self.dtype = torch.bfloat16


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,off", [(4, 0), (132, 4), (1536, 8), (1030, 0), (256, 3)])
@pytest.mark.parametrize("lens", [(1, 2, 3), (500, 13), (1, 1021, 5)])
def test_mixes_of_neighbouring_rows(cuda_kernels, dtype, C, off, lens):
    g = torch.Generator().manual_seed(C + sum(lens))
    x, mu, state = torch.randn(sum(lens), C, generator=g), torch.rand(5, C, generator=g), torch.randn(4, off + C, generator=g)
    slots = [2, 0, 3][:len(lens)]
    before = torch.cat([x[:1], x[:-1]]).double()
    at = 0
    for n, s in zip(lens, slots):
        before[at] = state[s, off:].double()
        at += n
    want = x.double() + (before - x.double()) * mu.double()[:, None]
    got = cuda_kernels.token_shift_mix(x.to(DEV), mu.to(DEV), state.to(DEV), off, _Ctx([(0, n) for n in lens], slots, DEV), dtype)
    _close(got, want, dtype)


@pytest.mark.parametrize("rank,ld,col0", [(8, 8, 0), (256, 320, 0), (512, 528, 16), (520, 520, 0), (1536, 1856, 0), (2048, 2048, 0), (2056, 2056, 0),
                                          (100, 100, 0), (256, 324, 4)])
def test_normed_columns(cuda_kernels, rank, ld, col0):
    g = torch.Generator().manual_seed(rank)
    rows, w = torch.randn(37, ld, generator=g).to(torch.bfloat16), 1 + 0.2 * torch.randn(rank, generator=g)
    x = rows.double()[:, col0:col0 + rank]
    want = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    _close(cuda_kernels.rmsnorm_columns(rows.to(DEV), col0, rank, w.to(DEV), 1e-6), want, torch.bfloat16)


@pytest.mark.parametrize("rot,used,interleaved", [(64, 64, True), (64, 64, False), (64, 32, True), (48, 16, False), (8, 8, False), (72, 72, True)])
@pytest.mark.parametrize("heads,lat", [(1, 256), (12, 256), (13, 40)])
def test_turned_latents(cuda_kernels, rot, used, interleaved, heads, lat):
    from types import SimpleNamespace
    g = torch.Generator().manual_seed(rot * 7 + heads)
    spans, slots, dim, page = [(5, 3), (0, 150)], (1, 0), 64, 16
    T = 153
    rows, q = torch.randn(T, lat + rot, generator=g).to(torch.bfloat16), torch.randn(T, heads * (dim + rot), generator=g).to(torch.bfloat16)
    w, freq = 1 + 0.2 * torch.randn(lat, generator=g), 10.0 ** (-4 * torch.arange(used // 2) / max(1, used // 2))
    ctx = _Ctx(spans, slots, DEV)
    table = torch.arange(20, dtype=torch.int32, device=DEV).view(2, 10)
    kv = torch.zeros(20, 1, 1, page, lat + rot, dtype=torch.bfloat16, device=DEV)
    rotary = SimpleNamespace(rotary_dim=used, interleaved=interleaved, magnitude=0.75, inv_freq=freq.to(DEV))
    turned = cuda_kernels.latent_rope_append(rows.to(DEV), 0, lat, rot, w.to(DEV), 1e-6, q.to(DEV), heads, dim, rotary, ctx,
                                             SimpleNamespace(kv=kv, block_table=table, writes=True, page_size=page))

    def turn(x):                                             # [T, n, rot]
        ang = (ctx.positions.cpu().float()[:, None] * freq).double()[:, None]
        a, b = (x[..., 0:used:2], x[..., 1:used:2]) if interleaved else (x[..., :used // 2], x[..., used // 2:used])
        c, s = 0.75 * ang.cos(), 0.75 * ang.sin()
        lo, hi = a * c - b * s, b * c + a * s
        return torch.cat((torch.stack((lo, hi), -1).flatten(-2) if interleaved else torch.cat((lo, hi), -1), x[..., used:]), -1)
    want = q.double().view(T, heads, dim + rot).clone()
    want[..., dim:] = turn(want[..., dim:])
    _close(turned, want.view(T, -1), torch.bfloat16)
    x = rows.double()
    row = torch.cat((x[:, :lat] * torch.rsqrt(x[:, :lat].square().mean(-1, keepdim=True) + 1e-6) * w.double(), turn(x[:, None, lat:])[:, 0]), -1)
    pos, slot = ctx.positions.cpu().long(), torch.tensor([1] * 3 + [0] * 150)
    held = kv.cpu().view(20, page, -1)[table.cpu()[slot, pos // page].long(), pos % page]
    _close(held, row, torch.bfloat16)


@pytest.mark.parametrize("rank", [8, 256, 264, 512, 520, 1536, 2040, 2048])
def test_a_normed_row_has_its_bits_wherever_it_lies(cuda_kernels, rank):
    """Rows on 16-byte boundaries and the same rows off them: one order of sums.  (700 rows: a sum in another order rounds some of their
    numbers differently.)"""
    g = torch.Generator().manual_seed(rank)
    rows, w = torch.randn(700, rank, generator=g).to(torch.bfloat16), (1 + 0.2 * torch.randn(rank, generator=g)).to(DEV)
    off = torch.zeros(700, rank + 1, dtype=torch.bfloat16)
    off[:, 1:] = rows
    assert torch.equal(cuda_kernels.rmsnorm_columns(rows.to(DEV), 0, rank, w, 1e-6), cuda_kernels.rmsnorm_columns(off.to(DEV), 1, rank, w, 1e-6))


@pytest.mark.parametrize("rot,used,interleaved", [(0, 0, False), (64, 64, True), (64, 32, False), (8, 2, False)])
@pytest.mark.parametrize("lat", [8, 256, 504, 512])
def test_a_turned_latent_has_its_bits_wherever_it_lies(cuda_kernels, rot, used, interleaved, lat):
    from types import SimpleNamespace
    g = torch.Generator().manual_seed(rot + lat)
    T, heads, dim, page = 700, 5, 64, 16
    rows, q = torch.randn(T, lat + rot, generator=g).to(torch.bfloat16), torch.randn(T, heads * (dim + rot), generator=g).to(torch.bfloat16)
    off = torch.zeros(T, lat + rot + 1, dtype=torch.bfloat16)
    off[:, 1:] = rows
    w, freq = (1 + 0.2 * torch.randn(lat, generator=g)).to(DEV), (10.0 ** (-4 * torch.arange(used // 2) / max(1, used // 2))).to(DEV)
    ctx = _Ctx([(31, T)], [0], DEV)
    table = torch.arange(46, dtype=torch.int32, device=DEV).view(1, 46)
    rotary = SimpleNamespace(rotary_dim=used, interleaved=interleaved, magnitude=0.75, inv_freq=freq) if used else None
    results = []
    for x, col0 in ((rows, 0), (off, 1)):
        kv = torch.zeros(46, 1, 1, page, lat + rot, dtype=torch.bfloat16, device=DEV)
        turned = cuda_kernels.latent_rope_append(x.to(DEV), col0, lat, rot, w, 1e-6, q.to(DEV), heads, dim, rotary, ctx,
                                                 SimpleNamespace(kv=kv, block_table=table, writes=True, page_size=page))
        results.append((turned, kv))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("T,groups,part", [(3, 9, 1), (5, 9, 20), (700, 40, 31), (700, 40, 32), (700, 40, 33), (41, 7, 63), (600, 40, 65), (600, 40, 127),
                                           (9, 3, 129), (2100, 10, 200), (2100, 10, 255), (4, 40, 16)])
@pytest.mark.parametrize("gate_first", [False, True])
def test_norm_and_gate_of_parts_of_any_size(cuda_kernels, T, groups, part, gate_first):
    """Sizes around those for which a lane has room; few rows, and so many that a warp takes several parts."""
    test_norm_and_gate(cuda_kernels, torch.bfloat16, T, groups, part, gate_first, "silu", 1)
    test_norm_and_gate(cuda_kernels, torch.float32, T, groups, part, gate_first, "sigmoid", 0)


@pytest.mark.parametrize("nq,nkv,d,T", [(64, 8, 128, 149), (40, 40, 128, 301), (65, 31, 128, 300), (12, 2, 128, 1333), (12, 2, 128, 2369), (28, 4, 128, 1777),
                                        (8, 8, 256, 593), (1, 1, 16, 9500)])
def test_turned_rows_have_their_bits_in_steps_of_any_size(cuda_kernels, nq, nkv, d, T):
    """One token a block and two, rows of one block an SM and of several: as in steps of 100 tokens, where every block has one."""
    from types import SimpleNamespace
    g = torch.Generator().manual_seed(T)
    qkv = torch.randn(T, (nq + 2 * nkv) * d, generator=g).to(torch.bfloat16).to(DEV)
    bias = torch.randn((nq + 2 * nkv) * d, generator=g).to(DEV)
    rotary = SimpleNamespace(rotary_dim=d, interleaved=False, magnitude=1.0, inv_freq=torch.rand(d // 2, generator=g).to(DEV))
    pages = -(-(T + 5) // 16)
    results = []
    for step in (T, 100):
        kv = torch.zeros(pages + 3, 2, nkv, 16, d, dtype=torch.bfloat16, device=DEV)
        table = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(1, -1).to(DEV)
        cache = SimpleNamespace(kv=kv, block_table=table, writes=True, page_size=16)
        out = []
        for t0 in range(0, T, step):
            ctx = _Ctx([(5 + t0, min(step, T - t0))], [0], DEV)
            ctx.extra_len = {"attn.prefill_tiles": 4, "attn.decode_rows": 0}
            out.append(cuda_kernels.rope_append(qkv[t0:t0 + step], bias, rotary, nq, nkv, d, ctx, cache))
        results.append((torch.cat(out), kv))
    if T % 100 >= 64 or T % 100 == 0:
        assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    else:                                                    # (fewer than 64 tokens: another kernel, with its own order of roundings)
        n = T - T % 100
        assert torch.equal(results[0][0][:n], results[1][0][:n])
        assert float((results[0][0].float() - results[1][0].float()).abs().max()) <= 2.0 ** -5
        assert float((results[0][1].float() - results[1][1].float()).abs().max()) <= 2.0 ** -5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("lens", [(1, 3, 1), (300,), (2049, 17)])
def test_a_convolution_has_its_bits_wherever_its_taps_lie(cuda_kernels, dtype, taps, lens):
    """Taps on a 16-byte boundary, read whole where there are four, and off it."""
    C, T = 264, sum(lens)
    g = torch.Generator().manual_seed(T + taps)
    x, w, st = torch.randn(T, C, generator=g).to(dtype).to(DEV), torch.randn(C, taps, generator=g).to(DEV), torch.randn(4, 1, taps - 1, C, generator=g)
    off = torch.zeros(C * taps + 1, device=DEV)
    off[1:] = w.reshape(-1)
    results = []
    for taken in (w, off[1:].view(C, taps)):
        state = st.to(DEV)
        out = cuda_kernels.short_conv(x, taken, taps, state, 0, _Ctx([(0, n) for n in lens], [2, 0, 3][:len(lens)], DEV))
        results.append((out, state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    want = torch.zeros(T, C, dtype=F64)
    at = 0
    for n, slot in zip(lens, [2, 0, 3]):
        rows = torch.cat([st[slot, 0].double(), x[at:at + n].double().cpu()])
        want[at:at + n] = x[at:at + n].double().cpu() + sum(rows[k:k + n] * w.double().cpu()[:, k] for k in range(taps))
        at += n
    _close(results[0][0], want, dtype)
