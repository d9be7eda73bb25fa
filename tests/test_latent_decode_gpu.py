"""Decoded tokens over cached latents of 256 (+ 64) numbers: lengths around tiles of 16 keys and whole stretches, windows that begin
inside a tile, more heads than a block takes, sinks and gates, pages longer than a tile; against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _setup(cuda_kernels, lens, rot, page, window, seed):
    from inferflux_b200.cache import CacheManager
    from inferflux_b200.config import ScheduleEntry
    from inferflux_b200.engine.batch import StepContext, StepEntry
    from inferflux_b200.parts import KVCacheSpec
    spec = KVCacheSpec(1, 256 + rot, window, planes=1)
    cache = CacheManager([(spec, None)], page_size=page, num_pages=sum(-(-n // page) for n in lens) + 3, max_seqs=len(lens),
                         max_seq_len=max(lens), dtype=BF, device=DEV)
    cache.groups[0].pool.copy_(torch.full_like(cache.groups[0].pool, float("nan")))     # what a page's former owner may have left
    g = torch.Generator().manual_seed(seed)
    kv, rows = cache.view(ScheduleEntry(0, 0)).kv, []
    for r, n in enumerate(lens):
        cache.add_request(r)
        cache.reserve(r, n)
        held, keys = cache.pages_of(r), torch.randn(n, 256 + rot, generator=g).to(BF)
        for b, p in held.items():
            part = keys[b * page:(b + 1) * page]
            kv[p, 0, 0, :len(part)] = part.to(DEV)
        rows.append(keys)
    ctx = StepContext.build(cuda_kernels, BF, torch.device(DEV), [StepEntry(r, [0], []) for r in range(len(lens))], [n - 1 for n in lens],
                            [cache.slot(r) for r in range(len(lens))], cache.drain_table_updates())
    for group, (index, pages) in zip(cache.groups, ctx.table_updates):
        cuda_kernels.scatter_i32(group.table, index, pages)
    return ctx, cache, cache.view(ScheduleEntry(0, 0)), rows, g


def _plain(ql, rows, window, scale, sinks, gate):
    """Weighted sums of latents [T, heads, 256]."""
    out = []
    for t, keys in enumerate(rows):
        k = keys.double()[max(0, len(keys) - window):] if window else keys.double()
        s = ql[t].double() @ k.T * scale
        if sinks is not None:
            s = torch.cat((s, sinks.double()[:, None]), -1)
        p = s.softmax(-1)[:, :len(k)]
        out.append(p @ k[:, :256] * (1.0 if gate is None else gate[t].double()[:, None]))
    return torch.stack(out)


@pytest.mark.parametrize("lens,heads,rot,page,window,extras", [
    ((1,), 12, 64, 16, None, False), ((15, 16, 17), 12, 64, 16, None, True), ((63, 64, 65, 1000), 28, 64, 16, None, False),
    ((129, 5000, 2), 12, 0, 32, None, True), ((700, 1, 333), 16, 64, 48, 100, True), ((401, 90, 16), 17, 0, 16, 33, False),
    ((20000,), 1, 64, 64, None, True), tuple([tuple(range(30, 1300, 20)), 12, 64, 16, None, False])])
def test_against_64_bits(cuda_kernels, lens, heads, rot, page, window, extras):
    ctx, cache, view, rows, g = _setup(cuda_kernels, lens, rot, page, window, len(lens) + heads)
    T, kw, scale = len(lens), 256 + rot, 0.2
    ql = torch.randn(T, heads, kw, generator=g).to(BF)
    sinks = torch.randn(heads, generator=g) if extras else None
    gate = torch.rand(T, heads, generator=g) if extras else None
    want = _plain(ql, rows, window, scale, sinks, gate)
    w = torch.eye(256, dtype=BF).repeat(heads, 1).to(DEV)                # queries and sums go through unchanged
    on = lambda t: None if t is None else t.to(DEV)
    if rot:
        from inferflux_b200.csrc.ops import TurnedQueries
        flat = torch.cat((ql[..., :256], torch.zeros(T, heads, rot, dtype=BF)), -1).to(DEV).reshape(T, -1)
        q = TurnedQueries(flat, ql.to(DEV).reshape(T, -1).clone())
    else:
        q = ql.to(DEV).reshape(T, -1)
    assert cuda_kernels.lib.ifx_latent_decode_supports(256, rot, page)
    stretch = cuda_kernels.lib.ifx_latent_decode_stretch(T, heads, int(ctx.max_kv_len if window is None else min(window, ctx.max_kv_len)))
    assert stretch % 64 == 0 and 64 <= stretch <= 1024
    got = cuda_kernels.latent_attention(q, w, w, on(sinks), heads, 256, 256, 256, window, scale, ctx, view, rot=rot, head_gate=on(gate))
    cuda_kernels.check_errors()
    got = got.view(T, heads, 256).double().cpu()
    # weights rounded to 8 bits, each on its own, over rows of size one; the sum's own rounding
    assert bool(torch.isfinite(got).all())
    assert float((got - want).abs().max()) <= 2.0 ** -7 * max(1.0, float(want.abs().max()))
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -8


@pytest.mark.parametrize("tiles", [False, True])                         # the kernel for decoded tokens, the tiles that share its merge
@pytest.mark.parametrize("keys", [40, 700])                              # one part, several
@pytest.mark.parametrize("what", ["query", "tile", "stretch", "outweighed"])
def test_what_is_not_finite_arrives_in_the_result(cuda_kernels, what, keys, tiles):
    """A query that is not a number, and keys that fill a warp's tile or a whole part, make their token's result no number, with
    the keys in one part or in several; so does an infinity of weight zero in a part that another part outweighs."""
    heads, rot, scale = 12, 64, 0.2
    ctx, cache, view, rows, g = _setup(cuda_kernels, (keys, keys), rot, 16, None, 7)
    ql = torch.randn(2, heads, 256 + rot, generator=g).to(BF)
    if what == "outweighed":
        ql[0, :, 7] = -1.0
    w = torch.eye(256, dtype=BF).repeat(heads, 1).to(DEV)
    from inferflux_b200.csrc.ops import TurnedQueries

    def run():
        flat = torch.cat((ql[..., :256], torch.zeros(2, heads, rot, dtype=BF)), -1).to(DEV).reshape(2, -1)
        before, cuda_kernels.latent_decode = cuda_kernels.latent_decode, not tiles
        try:
            got = cuda_kernels.latent_attention(TurnedQueries(flat, ql.to(DEV).reshape(2, -1).clone()), w, w, None, heads, 256, 256, 256,
                                                None, scale, ctx, view, rot=rot)
        finally:
            cuda_kernels.latent_decode = before
        cuda_kernels.check_errors()
        return got.view(2, heads, 256).float().cpu()

    def row(key, value):
        view.kv[cache.pages_of(0)[key // 16], 0, 0, key % 16] = value

    clean = run()
    assert bool(torch.isfinite(clean).all())
    fine = torch.ones_like(clean, dtype=torch.bool)
    if what == "query":
        ql[0, 3] = float("nan")
        fine[0, 3] = False
    elif what in ("tile", "stretch"):
        for key in range(16, 32) if what == "tile" else range(min(keys, 64)):
            row(key, float("nan"))
        fine[0] = False
    else:
        view.kv[cache.pages_of(0)[0], 0, 0, 5, 7] = float("inf")             # a score of -inf, a value of inf
        row(keys - 1, (8.0 * ql[0, 0].float()).to(BF).to(DEV))               # head 0: the last key is all there is
        fine[0] = False                                                  # (the product behind the sums spreads it over the columns)
    got = run()
    assert torch.equal(torch.isfinite(got), fine)
    assert torch.equal(got[1], clean[1])
