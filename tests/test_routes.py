"""Which kernels run when: the rules alone, without a GPU."""
import pytest
import torch

from inferflux_b200.csrc import CudaKernels


class _Table:
    """The rules of a kernel table that was never made."""
    chunk_scans = True
    CHUNK_SCAN_MIN_SPAN = CudaKernels.CHUNK_SCAN_MIN_SPAN
    stretches_pay, delta_stretches_pay = CudaKernels.stretches_pay, CudaKernels.delta_stretches_pay
    _long_spans = CudaKernels._long_spans
    _scans_by_chunks, _delta_by_chunks = CudaKernels._scans_by_chunks, CudaKernels._delta_by_chunks



class _Ctx:
    def __init__(self, lens):
        self.spans, self.num_requests, self.max_span = [(7, n) for n in lens], len(lens), max(lens)


ALL, NONE = (1, 0), False


@pytest.mark.parametrize("lens,scans,deltas", [
    ((2048,), ALL, ALL), ((127,), NONE, NONE), ((500, 400), ALL, ALL), ((512,) + (1,) * 31, (128, 1), (128, 1)),
    ((128,) + (1,) * 31, (128, 1), NONE), ((512, 1), ALL, ALL), ((200, 100), ALL, ALL), ((150, 71), ALL, ALL),
    ((512, 100, 80) + (1,) * 29, (128, 100), (128, 100)), ((200,) + (100,) * 30, NONE, NONE), ((128,) * 32, ALL, NONE), ((1,) * 32, NONE, NONE)])
def test_recurrences_by_stretches(lens, scans, deltas):
    """A decoded token is a stretch of its own, so what counts is stretches and what the scan would take, not the longest span alone:
    all spans by stretches, the long ones beside the scan for the others, or the scan."""
    table = _Table()
    ctx = _Ctx(lens)
    assert table._scans_by_chunks(torch.bfloat16, ctx, 12, 128, 128, constant=True) == scans
    assert table._delta_by_chunks(torch.bfloat16, ctx, sum(lens), 24, 64) == deltas
    assert not table._scans_by_chunks(torch.float32, ctx, 12, 128, 128) and not table._scans_by_chunks(torch.bfloat16, ctx, 12, 96, 128)
    short = [n for n in lens if n < 128]
    count = lambda spans: sum(-(-n // 64) for n in spans)
    assert table._long_spans(ctx) == (max(short, default=0), sum(short), len(short), count(short), count(n for n in lens if n >= 128))


def test_very_many_states_beside_the_shortest_long_span():
    table = _Table()
    for lens, way in (((128,) + (1,) * 63, NONE), ((192,) + (1,) * 63, (128, 1)), ((128,) + (1,) * 31, (128, 1))):
        assert table._scans_by_chunks(torch.bfloat16, _Ctx(lens), 28, 128, 128) == way


def test_a_constant_decay_with_small_keys_and_very_many_stretches_stays_with_the_scan():
    table = _Table()
    for lens, way in (((128,) * 32, False), ((256,) * 16, True), ((128,) * 16, True)):
        assert bool(table._scans_by_chunks(torch.bfloat16, _Ctx(lens), 28, 64, 128, constant=True)) == way
        assert table._scans_by_chunks(torch.bfloat16, _Ctx(lens), 28, 64, 128)


class _Counted(list):
    walks = 0

    def __iter__(self):
        self.walks += 1
        return super().__iter__()


def test_parts_of_the_prompt_attention_are_found_once_a_step_and_kind_of_layer():
    """Every layer asks; the spans are walked for the first one of a kind."""
    table = type("T", (), {"PREFILL_TILE": CudaKernels.PREFILL_TILE, "PREFILL_PART_TILES": CudaKernels.PREFILL_PART_TILES,
                           "prefill_parts": CudaKernels.prefill_parts, "_prefill_parts": CudaKernels._prefill_parts,
                           "attention_sections": CudaKernels.attention_sections})()

    def step(*spans):
        ctx = type("C", (), {})()
        ctx.spans, ctx.slots_host = _Counted(spans), list(range(len(spans)))
        ctx.extra_len = {k: len(v) for k, v in table.attention_sections(ctx).items()}
        ctx.spans.walks = 0
        return ctx

    ctx = step((1100, 300))
    assert [table.prefill_parts(ctx, 12, 0) for _ in range(5)] == [2] * 5 and ctx.spans.walks == 1
    assert table.prefill_parts(ctx, 12, 600) == 1 and table.prefill_parts(ctx, 12, 600) == 1 and ctx.spans.walks == 2
    ctx.spans = _Counted([(3000, 512)])                                         # another step's spans
    ctx.extra_len = {k: len(v) for k, v in table.attention_sections(ctx).items()}
    assert table.prefill_parts(ctx, 12, 0) == 6
    for spans, parts in ((((0, 900),), 1), (((0, 1152),), 2), (((5, 1), (9, 1)), 1)):     # eight tiles of keys stay whole
        assert table.prefill_parts(step(*spans), 12, 0) == parts
