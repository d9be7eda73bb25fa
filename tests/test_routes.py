"""Which kernels run when: the rules alone, without a GPU."""
import pytest
import torch

from inferflux_b200.csrc import CudaKernels


class _Table:
    """The rules of a kernel table that was never made."""
    chunk_scans = True
    CHUNK_SCAN_MIN_SPAN = CudaKernels.CHUNK_SCAN_MIN_SPAN
    stretches_pay, delta_stretches_pay = staticmethod(CudaKernels.stretches_pay), staticmethod(CudaKernels.delta_stretches_pay)
    _long_spans, _parting = CudaKernels._long_spans, CudaKernels._parting
    _scans_by_chunks, _delta_by_chunks = CudaKernels._scans_by_chunks, CudaKernels._delta_by_chunks

    class lib:
        ifx_chunk_scan_supports = ifx_delta_chunks_supports = staticmethod(lambda *a: 1)


class _Ctx:
    def __init__(self, lens):
        self.spans, self.num_requests, self.max_span = [(7, n) for n in lens], len(lens), max(lens)


SPANS = {"prompt": (2048,), "short prompt": (127,), "prompts": (500, 400), "portion and decoded": (512,) + (1,) * 31,
         "small portion and decoded": (128,) + (1,) * 31, "portion and a short span": (200, 100), "many": (128,) * 32, "decoded": (1,) * 32}


@pytest.mark.parametrize("kind,scans,deltas", [
    ("prompt", True, True), ("short prompt", False, False), ("prompts", True, True), ("portion and decoded", True, True),
    ("small portion and decoded", True, False), ("portion and a short span", False, False), ("many", True, False), ("decoded", False, False)])
def test_recurrences_by_stretches(kind, scans, deltas):
    """A decoded token is a stretch of its own, so what counts is stretches and what the scan would take, not the longest span alone."""
    table, lens = _Table(), SPANS[kind]
    ctx = _Ctx(lens)
    assert table._scans_by_chunks(torch.bfloat16, ctx, 12, 128, 128, constant=True) == scans
    assert table._delta_by_chunks(torch.bfloat16, ctx, sum(lens), 24, 64) == deltas
    assert not table._scans_by_chunks(torch.float32, ctx, 12, 128, 128)
    short = [n for n in lens if n < 128]
    assert table._parting(ctx) == (128, max(short, default=0))
    assert table._long_spans(ctx) == (max(short, default=0), sum(short), len(short), sum(-(-n // 64) for n in lens if n >= 128))


def test_a_constant_decay_with_small_keys_and_very_many_stretches_stays_with_the_scan():
    table = _Table()
    for lens, way in (((128,) * 32, False), ((256,) * 16, True), ((128,) * 16, True)):
        assert table._scans_by_chunks(torch.bfloat16, _Ctx(lens), 28, 64, 128, constant=True) == way
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
