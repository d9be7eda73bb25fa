"""Prompt portions over cached latents of 256 (+ 64) numbers on tcgen05: spans around tiles of 128 rows and 128 keys, context in
front, windows, sinks, gates, keys cut into parts, numbers that are not finite; against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _setup(cuda_kernels, spans, rot, page, window, seed):
    """`spans`: (tokens of context, new tokens).  Returns the step context, the cache's view, every request's rows."""
    from inferflux_b200.cache import CacheManager
    from inferflux_b200.config import ScheduleEntry
    from inferflux_b200.engine.batch import StepContext, StepEntry
    from inferflux_b200.parts import KVCacheSpec
    spec = KVCacheSpec(1, 256 + rot, window, planes=1)
    cache = CacheManager([(spec, None)], page_size=page, num_pages=sum(-(-(c + n) // page) for c, n in spans) + 3, max_seqs=len(spans),
                         max_seq_len=max(c + n for c, n in spans), dtype=BF, device=DEV)
    cache.groups[0].pool.fill_(float("nan"))                             # what a page's former owner may have left
    g = torch.Generator().manual_seed(seed)
    kv, rows = cache.view(ScheduleEntry(0, 0)).kv, []
    for r, (c, n) in enumerate(spans):
        cache.add_request(r)
        cache.reserve(r, c + n)
        keys = torch.randn(c + n, 256 + rot, generator=g).to(BF)
        for b, p in cache.pages_of(r).items():
            part = keys[b * page:(b + 1) * page]
            kv[p, 0, 0, :len(part)] = part.to(DEV)
        rows.append(keys)
    ctx = StepContext.build(cuda_kernels, BF, torch.device(DEV), [StepEntry(r, [0] * n, []) for r, (_c, n) in enumerate(spans)],
                            [c for c, _n in spans], [cache.slot(r) for r in range(len(spans))], cache.drain_table_updates())
    for group, (index, pages) in zip(cache.groups, ctx.table_updates):
        cuda_kernels.scatter_i32(group.table, index, pages)
    return ctx, cache, cache.view(ScheduleEntry(0, 0)), rows, g


def _plain(ql, spans, rows, window, scale, sinks, gate):
    out, at = [], 0
    for (c, n), keys in zip(spans, rows):
        k = keys.double()
        pos, key = torch.arange(c, c + n)[:, None], torch.arange(c + n)[None]
        hidden = key > pos
        if window:
            hidden |= key < pos - window + 1
        s = torch.einsum("thd,kd->htk", ql[at:at + n].double(), k) * scale
        s = s.masked_fill(hidden, float("-inf"))
        if sinks is not None:
            s = torch.cat((s, sinks.double()[:, None, None].expand(-1, n, 1)), -1)
        p = s.softmax(-1)[..., :c + n]
        out.append(torch.einsum("htk,kd->thd", p, k[:, :256]))
        at += n
    out = torch.cat(out)
    return out if gate is None else out * gate.double()[..., None]


def _run(cuda_kernels, ctx, view, ql, heads, rot, window, scale, sinks, gate):
    on = lambda t: None if t is None else t.to(DEV)
    T = ql.shape[0]
    w = torch.eye(256, dtype=BF).repeat(heads, 1).to(DEV)                # queries and sums go through unchanged
    if rot:
        from inferflux_b200.csrc.ops import TurnedQueries
        flat = torch.cat((ql[..., :256], torch.zeros(T, heads, rot, dtype=BF)), -1).to(DEV).reshape(T, -1)
        q = TurnedQueries(flat, ql.to(DEV).reshape(T, -1).clone())
    else:
        q = ql.to(DEV).reshape(T, -1)
    got = cuda_kernels.latent_attention(q, w, w, on(sinks), heads, 256, 256, 256, window, scale, ctx, view, rot=rot, head_gate=on(gate))
    cuda_kernels.check_errors()
    return got.view(T, heads, 256).double().cpu()


@pytest.mark.parametrize("spans,heads,rot,page,window,extras", [
    ([(0, 6)], 12, 64, 16, None, False), ([(0, 64), (0, 65)], 12, 64, 16, None, True), ([(0, 11), (117, 300)], 12, 0, 32, None, True),
    ([(1000, 40)], 28, 64, 16, None, True), ([(0, 700)], 16, 64, 48, 100, True), ([(90, 129), (500, 8)], 17, 0, 16, 33, False),
    ([(127, 257)], 1, 64, 64, None, True), ([(5000, 70)], 1, 64, 16, 2000, False), ([(0, 1500), (3, 128)], 12, 64, 16, None, False)])
def test_against_64_bits(cuda_kernels, spans, heads, rot, page, window, extras):
    ctx, cache, view, rows, g = _setup(cuda_kernels, spans, rot, page, window, len(spans) + heads)
    T, scale = sum(n for _c, n in spans), 0.2
    assert min(n for _c, n in spans) * heads >= cuda_kernels.LATENT_PROMPT_MIN_ROWS
    assert cuda_kernels.lib.ifx_latent_prompt_supports(256, rot, page)
    ql = torch.randn(T, heads, 256 + rot, generator=g).to(BF)
    sinks = torch.randn(heads, generator=g) if extras else None
    gate = torch.rand(T, heads, generator=g) if extras else None
    want = _plain(ql, spans, rows, window, scale, sinks, gate)
    got = _run(cuda_kernels, ctx, view, ql, heads, rot, window, scale, sinks, gate)
    # weights rounded to 8 bits, each on its own, over rows of size one; the sum's own rounding
    assert bool(torch.isfinite(got).all())
    assert float((got - want).abs().max()) <= 2.0 ** -7 * max(1.0, float(want.abs().max()))
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -8


def test_scores_that_grow_far_beyond_the_first_ones(cuda_kernels):
    """The reference maximum moves in every tile: the sums are scaled again and again."""
    spans, heads, rot, scale = [(0, 900)], 12, 64, 1.0
    ctx, cache, view, rows, g = _setup(cuda_kernels, spans, rot, 16, None, 3)
    size = torch.linspace(0.01, 3.0, 900)[:, None]
    rows[0].copy_((rows[0].float() * size).to(BF))
    for b, p in cache.pages_of(0).items():
        part = rows[0][b * 16:(b + 1) * 16]
        view.kv[p, 0, 0, :len(part)] = part.to(DEV)
    ql = torch.randn(900, heads, 256 + rot, generator=g).to(BF)
    want = _plain(ql, spans, rows, None, scale, None, None)
    got = _run(cuda_kernels, ctx, view, ql, heads, rot, None, scale, None, None)
    assert float((got - want).abs().max()) <= 2.0 ** -6 * float(want.abs().max())


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("window", [None, 60])
def test_a_row_that_is_not_finite_reaches_those_who_see_it(cuda_kernels, value, window):
    spans, heads, rot, scale, at = [(30, 400)], 12, 64, 0.2, 200
    ctx, cache, view, rows, g = _setup(cuda_kernels, spans, rot, 16, window, 4)
    ql = torch.randn(400, heads, 256 + rot, generator=g).to(BF)
    clean = _run(cuda_kernels, ctx, view, ql, heads, rot, window, scale, None, None)
    view.kv[cache.pages_of(0)[at // 16], 0, 0, at % 16, 7] = value
    got = _run(cuda_kernels, ctx, view, ql, heads, rot, window, scale, None, None)
    sees = torch.arange(30, 430) >= at
    if window:
        sees &= torch.arange(30, 430) < at + window
    assert torch.equal(got[~sees], clean[~sees])
    assert not bool(torch.isfinite(got[sees]).all(-1).any())


@pytest.mark.parametrize("tiles", [False, True])                         # tcgen05, the mma.sync tiles that share its merge
@pytest.mark.parametrize("context", [0, 1000])                           # one part, several
@pytest.mark.parametrize("what", ["query", "keys"])
def test_what_is_not_a_number_arrives_in_the_result(cuda_kernels, what, context, tiles):
    """A query that is not a number, and keys that fill the first part, make the result of those who see them no number, with the
    keys in one part or in several."""
    spans, heads, rot, scale, at = [(context, 40)], 12, 64, 0.2, 17
    ctx, cache, view, rows, g = _setup(cuda_kernels, spans, rot, 16, None, 8)
    ql = torch.randn(40, heads, 256 + rot, generator=g).to(BF)
    before, cuda_kernels.latent_prompt = cuda_kernels.latent_prompt, not tiles
    try:
        clean = _run(cuda_kernels, ctx, view, ql, heads, rot, None, scale, None, None)
        bad = torch.zeros(40, heads, dtype=torch.bool)
        if what == "query":
            ql[at, 3] = float("nan")
            bad[at, 3] = True
        else:
            for key in range(512 if context else 1):                     # with context: all that the first parts hold
                view.kv[cache.pages_of(0)[key // 16], 0, 0, key % 16] = float("nan")
            bad[:] = True
        got = _run(cuda_kernels, ctx, view, ql, heads, rot, None, scale, None, None)
    finally:
        cuda_kernels.latent_prompt = before
    assert bool(torch.isfinite(clean).all())
    assert torch.equal(torch.isfinite(got), (~bad)[..., None].expand_as(got))
    assert torch.equal(got[~bad], clean[~bad])


@pytest.mark.parametrize("scale", [0.0, -0.2])
def test_a_scale_that_is_not_positive_keeps_the_tiles(cuda_kernels, scale):
    """The running maximum of the tcgen05 kernel is of the scores before they are scaled."""
    spans, heads, rot = [(30, 70)], 12, 64
    ctx, cache, view, rows, g = _setup(cuda_kernels, spans, rot, 16, None, 9)
    ql = torch.randn(70, heads, 256 + rot, generator=g).to(BF)
    want = _plain(ql, spans, rows, None, scale, None, None)
    got = _run(cuda_kernels, ctx, view, ql, heads, rot, None, scale, None, None)
    assert float((got - want).abs().max()) <= 2.0 ** -7 * max(1.0, float(want.abs().max()))
