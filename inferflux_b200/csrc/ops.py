"""The kernel table of the product path: every operation of a step as a call into
the hand-written sm_100a library (plus cuBLAS for the bfloat16 matrix products,
where the reference uses it too).

There is no CPU path and no library model code here: making a `CudaKernels`
without a CUDA device, or without being able to build or load the library, raises.
Tensors are passed as raw device pointers (host_call.cpp) on torch's current stream.  What a call costs the host
matters where a layer's kernels are short: sizes go to `torch.empty` one by one (as a tuple they
take a microsecond more), and messages with values in them are made when something is wrong.
"""
from __future__ import annotations

import ctypes
import os

import torch

from .build import BuildError, HostLibrary, load_library

_DT = {torch.float32: 0, torch.bfloat16: 1}
_MISALIGNED = -3             # what the kernels of long spans say of rows off a 16-byte boundary, before they touch anything
_DECAYS = {"sigmoid_root": 0, "softplus_step": 1, "constant": 2}

_ERRORS = {-1: "a size or option the kernel does not take", -2: "unknown dtype",
           -3: "a pointer or stride breaks an alignment rule", -4: "a size beyond the kernel's stated maximum"}


class KernelError(RuntimeError):
    pass


class ScaledRows:
    """Rows of a norm without its row scale: `pre` = x * w in the run's dtype and `sumsq`
    [rows, chunks] float32, the chunks' sums of x^2.  The true rows are
    pre * rsqrt(sum(sumsq[row]) / hidden + eps); a matrix product that takes them applies that
    per-row factor to its accumulator.  `CudaKernels.materialize_rows` gives the plain tensor."""

    def __init__(self, pre: torch.Tensor, sumsq: torch.Tensor, eps: float):
        self.pre, self.sumsq, self.eps = pre, sumsq, float(eps)

    @property
    def shape(self):
        return self.pre.shape

    @property
    def dtype(self):
        return self.pre.dtype


class PartialSum:
    """The result of a matrix product whose K range was split over thread blocks:
    float32 partial sums [splits, rows, cols] that the consuming kernel adds, in split
    order, in the same pass in which it does its own work (residual add and norm, bias
    and rotation).  `CudaKernels.materialize` gives the plain tensor."""

    def __init__(self, parts: torch.Tensor, dtype: torch.dtype):
        self.parts = parts
        self.dtype = dtype                       # the dtype the sum stands for

    @property
    def shape(self):
        return self.parts.shape[1:]

    @property
    def splits(self) -> int:
        return self.parts.shape[0]


# The current stream's handle of the current device, asked for at every launch: torch's own accessors
# when they are there (plain integers, a fraction of a microsecond), else through the Stream object
# (several microseconds).
_RAW_STREAM = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_RAW_DEVICE = getattr(torch._C, "_cuda_getDevice", None)


def _stream():
    if _RAW_STREAM is not None and _RAW_DEVICE is not None:
        return _RAW_STREAM(_RAW_DEVICE())
    return torch.cuda.current_stream().cuda_stream


def _check(rc: int, what: str) -> None:
    if rc == 0:
        return
    if rc < 0:
        raise KernelError(f"{what}: refused ({_ERRORS.get(rc, rc)})")
    if rc >= 1000:
        raise KernelError(f"{what}: cuBLAS status {rc - 1000}")
    raise KernelError(f"{what}: CUDA error {rc}")


def _need(cond: bool, msg: str) -> None:
    if not cond:
        raise KernelError(msg)


_I, _F, _P, _LL = ctypes.c_int, ctypes.c_float, ctypes.c_void_p, ctypes.c_longlong       # of the structures below


class TurnedQueries:
    """Query rows [T, heads (dim + rot)] whose turned parts already lie in `latent`, the rows of queries in latent
    space [T, heads (rank + rot)] that the tiled latent attention reads."""
    __slots__ = ("rows", "latent")

    def __init__(self, rows, latent):
        self.rows, self.latent = rows, latent


class _StepArgs(ctypes.Structure):
    """IfxStepArgs of csrc/layer_forward.cu: one step's batch, the same for every layer."""
    _fields_ = ([(n, _I) for n in ("T", "num_decode", "num_tiles", "max_kv_len")]
                + [(n, _P) for n in ("positions", "token_req", "req_slot", "decode_rows", "decode_meta", "prefill_tiles",
                                     "norm_sumsq", "norm_tickets", "error_flag")]
                + [(n, _I) for n in ("skinny_max_rows", "swiglu_tiles", "swiglu_tiles_max_k", "tensor_core_prefill",
                                     "overlap_attention", "pad0")])


class _LayerArgs(ctypes.Structure):
    """IfxLayerArgs: one layer's sizes, constants, weights and cache."""
    _fields_ = ([(n, _I) for n in ("hidden", "inter", "nq", "nkv", "d", "window", "rot", "interleaved")]
                + [(n, _F) for n in ("scale", "eps_in", "eps_post")] + [("write_cache", _I)]
                + [(n, _P) for n in ("norm_in_w", "norm_post_w", "b_qkv", "inv_freq", "w_qkv", "w_o", "w_gate_up", "w_down",
                                     "kv_pool", "block_table")]
                + [(n, _I) for n in ("max_blocks", "page_size", "num_pages", "pad0")])


class _LayerIO(ctypes.Structure):
    """IfxLayerIO: what changes from call to call, and what comes back."""
    _fields_ = [("x", _P), ("pending_tensor", _P), ("pending_parts", _P), ("pending_splits", _I), ("parity", _I),
                ("ws", _P), ("ws_bytes", _LL), ("out_tensor", _P), ("out_parts", _P), ("out_splits", _I),
                ("launches", _I), ("library_calls", _I), ("prefill_parts", _I), ("least_decode_splits", _I), ("pad0", _I)]


class CudaKernels:
    """Kernel table on one CUDA device."""

    name = "cuda-sm100a"
    fuses_single_token_conv = True     # postnorm_add takes a short convolution for steps of single tokens

    def __init__(self, device="cuda"):
        if not torch.cuda.is_available():
            raise BuildError("no CUDA device: the engine has no CPU path")
        self.device = torch.device(device)
        self.lib = HostLibrary(
                  load_library(),
                  ("ifx_embed", "ifx_rmsnorm", "ifx_silu_mul", "ifx_residual_add", "ifx_gather_rows",
                   "ifx_scatter_i32", "ifx_rope_append", "ifx_attention_generic", "ifx_gemm_generic",
                   "ifx_gemm_cublas_bf16", "ifx_cublas_init", "ifx_argmax", "ifx_penalties", "ifx_logit_bias",
                   "ifx_sample", "ifx_sample_blocks", "ifx_attention_mma_supports", "ifx_attention_prefill_bf16",
                   "ifx_attention_prefill_tcgen05", "ifx_attention_prefill_tcgen05_supports", "ifx_attention_decode_max_splits",
                   "ifx_attention_decode_bf16", "ifx_gemm_skinny", "ifx_residual_add_partial",
                   "ifx_reduce_partial", "ifx_reduce_add_rmsnorm", "ifx_argmax_chunks", "ifx_relay_i32", "ifx_prenorm", "ifx_scale_rows",
                   "ifx_gemm_tcgen05", "ifx_postnorm_add_rmsnorm", "ifx_concat_cast", "ifx_xielu", "ifx_softcap",
                   "ifx_short_conv", "ifx_latent_norm_append", "ifx_latent_attention_generic", "ifx_latent_attention_mma",
                   "ifx_latent_attention_mma_supports", "ifx_gemm_cublas_bf16_batched", "ifx_gemm_skinny_act",
                   "ifx_attention_generic_ex", "ifx_norm_rope_append", "ifx_token_shift_mix", "ifx_cast_rows",
                   "ifx_wkv_scan", "ifx_moe_route", "ifx_moe_experts", "ifx_tanh_rows",
                   "ifx_attention_prefill_bf16_ex", "ifx_attention_decode_bf16_ex", "ifx_moe_sorted",
                   "ifx_attention_prefill_tcgen05_ex",
                   "ifx_groupnorm_stream", "ifx_residual_add_scaled", "ifx_gelu_mul_table", "ifx_embed_scaled", "ifx_scale_f32",
                   "ifx_delta_rule_scan", "ifx_latent_rope_append", "ifx_latent_attention_generic_rot", "ifx_moe_route_ex",
                   "ifx_moe_experts_ex", "ifx_latent_attention_mma_rot", "ifx_latent_attention_mma_supports_rot",
                   "ifx_moe_route_kind", "ifx_moe_choose", "ifx_moe_experts_glu", "ifx_norm_rope_append_ex",
                   "ifx_attention_generic_sink", "ifx_short_conv_ex", "ifx_decay_scan", "ifx_decay_scan_split", "ifx_bigram_add",
                   "ifx_rmsnorm_pair", "ifx_gate_mul", "ifx_gated_groupnorm", "ifx_pair_combine", "ifx_residual_add_vectors",
                   "ifx_attention_prefill_tcgen05_sink", "ifx_attention_prefill_bf16_sink", "ifx_attention_decode_bf16_sink",
                   "ifx_norm_of_sum", "ifx_row_norm_rope_append", "ifx_rotate_rows", "ifx_gated_scan", "ifx_decay_scan_rate",
                   "ifx_geglu_mul", "ifx_gemm_skinny_geglu", "ifx_gemm_tcgen05_geglu", "ifx_relu2", "ifx_silu_columns",
                   "ifx_chunk_scan_supports", "ifx_chunk_scan_takes_128", "ifx_chunk_decay_scan", "ifx_chunk_wkv_scan", "ifx_wkv_norm",
                   "ifx_latent_decode", "ifx_latent_decode_supports", "ifx_latent_decode_stretch",
                   "ifx_latent_prompt", "ifx_latent_prompt_supports", "ifx_delta_chunks_supports", "ifx_delta_chunks_scan",
                   "ifx_attention_prefill_tcgen05_parts", "ifx_gemm_f32_split", "ifx_swiglu_few", "ifx_gemm_f32_split_launches",
                   "ifx_set_shared_carveout", "ifx_set_pdl"),
                  ("ifx_delta_rule_scratch_floats", "ifx_chunk_scan_scratch_floats", "ifx_delta_chunks_scratch_floats",
                   "ifx_attention_prefill_tcgen05_parts_bytes", "ifx_gemm_f32_split_scratch", "ifx_moe_sorted_scratch",
                   "ifx_sample_scratch_bytes", "ifx_latent_attention_mma_workspace", "ifx_layer_workspace_bytes"))
        # long spans of a bfloat16 run's recurrences by stretches of 64 or 128 tokens (0: token after token, for comparisons)
        self.chunk_scans = os.environ.get("INFERFLUX_B200_CHUNK_SCANS", "1") != "0"
        self._latent_sizes = {}
        # latent attention on the tensor-core tiles (0: the per-token kernel, for comparisons)
        self.latent_tiles = os.environ.get("INFERFLUX_B200_LATENT_TILES", "1") != "0"
        # decoded tokens on the kernel made for them (0: the tiles of prompt portions, for comparisons)
        self.latent_decode = os.environ.get("INFERFLUX_B200_LATENT_DECODE", "1") != "0"
        # prompt portions on the tcgen05 kernel (0: the mma.sync tiles, for comparisons)
        self.latent_prompt = os.environ.get("INFERFLUX_B200_LATENT_PROMPT", "1") != "0"
        with torch.cuda.device(self.device):
            _check(self.lib.ifx_cublas_init(), "cublas init")
        if os.environ.get("INFERFLUX_B200_CARVEOUT", "") != "":    # for measurements: -1 leaves the split to the driver
            self.lib.ifx_set_shared_carveout(int(os.environ["INFERFLUX_B200_CARVEOUT"]))
        if os.environ.get("INFERFLUX_B200_PDL", "1") == "0":      # for measurements: no overlap of consecutive kernels
            self.lib.ifx_set_pdl(0)
        # prompt portions on the tcgen05 attention kernel (0: the mma.sync kernel, for comparisons)
        self.tensor_core_prefill = os.environ.get("INFERFLUX_B200_TCGEN05_ATTENTION", "1") != "0"
        # gate/up of prompt portions on the own tcgen05 tiles with the activation fused (0: cuBLAS + silu kernel)
        self.swiglu_tiles = os.environ.get("INFERFLUX_B200_SWIGLU_TILES", "1") != "0"
        self.launches = 0            # kernels of this library launched so far
        self.library_calls = 0       # cuBLAS products called so far
        # scratch of the many-block reduce + norm: sums of squares per (row, chunk), a ticket per row
        self._norm_sumsq = torch.zeros(128 * 64, dtype=torch.float32, device=self.device)
        self._norm_tickets = torch.zeros(128, dtype=torch.int32, device=self.device)
        self._sample_scratch, self._sample_capacity = None, 0   # zeroed once; the sampling kernels leave it zero
        self._argmax_val = torch.zeros(256 * 32, dtype=torch.float32, device=self.device)
        self._argmax_idx = torch.zeros(256 * 32, dtype=torch.int32, device=self.device)
        self._argmax_tickets = torch.zeros(256, dtype=torch.int32, device=self.device)
        self.error_flag = torch.zeros(1, dtype=torch.int32, device=self.device)   # set by a kernel whose bounded wait ran out
        # whole layers from native code (0: every part launches its kernels from Python, the general way)
        self.native_layers = os.environ.get("INFERFLUX_B200_NATIVE_LAYER", "1") != "0"
        # in a natively run layer of a mixed step, the two attention kernels side by side on two streams
        self.overlap_attention = os.environ.get("INFERFLUX_B200_ATTENTION_OVERLAP", "1") != "0"
        self.lib.ifx_layer_forward.restype = ctypes.c_int          # (takes structures: a ctypes function)
        self._layer_ws, self._layer_ws_all, self._layer_views = None, [], {}
        self._layer_io = _LayerIO()
        self._layer_io_ref = ctypes.byref(self._layer_io)
        self._layer_parity = 0
        self.native_layer_calls = 0

    # ------------------------------------------------------------- elementwise
    def embed(self, table, token_ids, vocab, scale=1.0):
        T, H = token_ids.numel(), table.shape[1]
        out = torch.empty(T, H, dtype=torch.float32, device=table.device)
        if scale != 1.0:
            _check(self.lib.ifx_embed_scaled(table, token_ids, out, T, H, int(vocab), float(scale),
                                             _DT[table.dtype], _stream()), "embed")
            self.launches += 1
            return out
        _check(self.lib.ifx_embed(table, token_ids, out, T, H, int(vocab), _DT[table.dtype],
                                  _stream()), "embed")
        self.launches += 1
        return out

    def rmsnorm(self, x, w, eps, out_dtype, groups=1):
        _need(x.dtype == torch.float32 and w.dtype == torch.float32, "rmsnorm: x and w must be float32")
        T, H = x.shape
        out = torch.empty(T, H, dtype=out_dtype, device=x.device)
        if groups > 1:
            _need(x.is_contiguous() and H % groups == 0, "rmsnorm: the groups must cut a contiguous row evenly")
            _check(self.lib.ifx_groupnorm_stream(
                x, None, None, 0.0, w, float(eps), int(groups), out,
                None, T, H, 0, _DT[out_dtype], 1, None, 0, None, 0, None,
                None, _stream()), "rmsnorm (groups)")
            self.launches += 1
            return out
        _check(self.lib.ifx_rmsnorm(x, None, w, out, T, H, float(eps), 0,
                                    _DT[out_dtype], _stream()), "rmsnorm")
        self.launches += 1
        return out

    def add_rmsnorm(self, x, delta, w, eps, out_dtype):
        """x += delta (in place), then the norm of the sum.  `delta` is a tensor in the run's
        dtype or a PartialSum, whose slices are added in the same pass."""
        _need(x.dtype == torch.float32 and w.dtype == torch.float32, "add_rmsnorm: x and w must be float32")
        T, H = x.shape
        out = torch.empty(T, H, dtype=out_dtype, device=x.device)
        if isinstance(delta, PartialSum):
            _need(tuple(delta.shape) == (T, H), "add_rmsnorm: partial sums do not match x")
            chunks = -(-H // 512)
            if T <= self._norm_tickets.numel() and T * chunks <= self._norm_sumsq.numel():
                _check(self.lib.ifx_reduce_add_rmsnorm(
                    x, delta.parts, w, out, T, H, float(eps), delta.splits,
                    self._norm_sumsq, self._norm_tickets, _DT[out_dtype], _stream()), "reduce_add_rmsnorm")
                self.launches += 1
                return out
            src, splits = delta.parts, delta.splits
        else:
            _need(delta.dtype == out_dtype and delta.shape == x.shape, "add_rmsnorm: delta must match x and the dtype")
            src, splits = delta, 0
        _check(self.lib.ifx_rmsnorm(x, src, w, out, T, H, float(eps), splits,
                                    _DT[out_dtype], _stream()), "add_rmsnorm")
        self.launches += 1
        return out

    def prenorm(self, x, delta, w, eps, out_dtype):
        """The norm for a consumer that takes ScaledRows (x += delta first, as add_rmsnorm).
        Few bfloat16 rows: one pass that leaves x * w and per-chunk sums of squares, the row scale
        being applied by the matrix product that follows.  Otherwise the plain normed tensor."""
        T, H = x.shape
        if out_dtype != torch.bfloat16 or T > self.SKINNY_MAX_ROWS or H % 8:
            return self.rmsnorm(x, w, eps, out_dtype) if delta is None else self.add_rmsnorm(x, delta, w, eps, out_dtype)
        pre = torch.empty(T, H, dtype=out_dtype, device=x.device)
        sumsq = torch.empty(T, -(-H // 512), dtype=torch.float32, device=x.device)
        if isinstance(delta, PartialSum):
            _need(tuple(delta.shape) == (T, H), "prenorm: partial sums do not match x")
            src, splits = delta.parts, delta.splits
        else:
            _need(delta is None or (delta.dtype == out_dtype and delta.shape == x.shape), "prenorm: delta must match x")
            src, splits = delta, 0
        _check(self.lib.ifx_prenorm(x, src, w, pre, sumsq, T, H, splits, _DT[out_dtype],
                                    _stream()), "prenorm")
        self.launches += 1
        return ScaledRows(pre, sumsq, eps)

    def materialize_rows(self, h):
        """A plain tensor from what `prenorm` returned."""
        if not isinstance(h, ScaledRows):
            return h
        T, H = h.shape
        out = torch.empty(T, H, dtype=h.dtype, device=h.pre.device)
        _check(self.lib.ifx_scale_rows(h.pre, h.sumsq, out, T, H, float(h.eps),
                                       _DT[h.dtype], _stream()), "scale_rows")
        self.launches += 1
        return out

    def residual_add(self, x, delta):
        T, H = x.shape
        if isinstance(delta, PartialSum):
            _check(self.lib.ifx_residual_add_partial(x, delta.parts, T, H, delta.splits, _stream()),
                   "residual_add")
        else:
            _check(self.lib.ifx_residual_add(x, delta, T, H, _DT[delta.dtype], _stream()), "residual_add")
        self.launches += 1

    def materialize(self, value, bias=None):
        """A plain tensor from what `linear(..., allow_partial=True)` returned."""
        if not isinstance(value, PartialSum):
            return value if bias is None else value + bias.to(value.dtype)
        T, N = value.shape
        out = torch.empty(T, N, dtype=value.dtype, device=value.parts.device)
        _check(self.lib.ifx_reduce_partial(value.parts, bias, out, T, N, value.splits,
                                           _DT[value.dtype], _stream()), "reduce_partial")
        self.launches += 1
        return out

    def silu_mul(self, gate_up):
        T, two_i = gate_up.shape
        out = torch.empty(T, two_i // 2, dtype=gate_up.dtype, device=gate_up.device)
        _check(self.lib.ifx_silu_mul(gate_up, out, T, two_i // 2, _DT[gate_up.dtype], _stream()),
               "silu_mul")
        self.launches += 1
        return out

    def gather_rows(self, x, rows):
        R, H = rows.numel(), x.shape[1]
        out = torch.empty(R, H, dtype=torch.float32, device=x.device)
        _check(self.lib.ifx_gather_rows(x, rows, out, R, H, x.shape[0], _stream()), "gather_rows")
        self.launches += 1
        return out

    def scatter_i32(self, table, index, value):
        n = index.numel()
        if n:
            _check(self.lib.ifx_scatter_i32(table, index, value, n, table.numel(), _stream()),
                   "scatter_i32")
            self.launches += 1

    def relay_i32(self, dst, dst_index, src, src_index):
        n = dst_index.numel()
        if n:
            _check(self.lib.ifx_relay_i32(dst, dst_index, src, src_index, n, dst.numel(),
                                          src.numel(), _stream()), "relay_i32")
            self.launches += 1

    # ------------------------------------------------------------------ linear
    # The weight-streaming kernel takes up to 256 rows; in a whole step it beats cuBLAS up to about 160
    # (measured at the 7B shape: 4.5 against 4.9 ms at 129 rows, 5.2 against 5.0 ms at 192).
    SKINNY_MAX_ROWS = 160

    def linear(self, a, w, bias=None, out_dtype=None, allow_partial=False):
        """out[T, N] = a[T, K] . w[N, K]^T (+ bias), float32 accumulation.  float32 runs use
        the CUDA-core product, or for large weights operands in parts on the tensor cores (`float32_by_parts`).  bfloat16 runs
        with up to SKINNY_MAX_ROWS rows use the tcgen05 weight-streaming kernel; with `allow_partial` a narrow product is split over K and comes back as a
        PartialSum for a consumer that adds the slices itself.  More rows go to cuBLAS."""
        rows = a if isinstance(a, ScaledRows) else None
        if rows is not None:
            a = rows.pre
        if a.dtype != w.dtype:                             # (messages with values in them are made when they are needed)
            raise KernelError(f"linear: activations are {a.dtype}, weights {w.dtype}")
        _need(a.is_contiguous() and w.is_contiguous(), "linear: operands must be contiguous")
        T, K = a.shape
        N = w.shape[0]
        if w.shape[1] != K:
            raise KernelError(f"linear: inner sizes differ ({K} vs {w.shape[1]})")
        out_dtype = out_dtype or a.dtype
        if T == 0:
            return torch.empty(T, N, dtype=out_dtype, device=a.device)
        if rows is not None and not (T <= self.SKINNY_MAX_ROWS and K % 8 == 0 and w.data_ptr() % 16 == 0):
            a, rows = self.materialize_rows(rows), None
        if a.dtype == torch.float32:
            _need(out_dtype == torch.float32, "linear: a float32 product gives float32")
            out = torch.empty(T, N, dtype=out_dtype, device=a.device)
            if self.float32_by_parts(N, K) and (a.data_ptr() | w.data_ptr()) % 16 == 0:
                room = self.lib.ifx_gemm_f32_split_scratch(T, N, K)
                scratch = torch.empty(room, dtype=torch.uint8, device=a.device)
                _check(self.lib.ifx_gemm_f32_split(a, w, bias, out, T, N, K, scratch, room,
                                                   self.error_flag, _stream()), "gemm (float32 by parts)")
                self.launches += self.lib.ifx_gemm_f32_split_launches(T, N, K)
                return out
            _check(self.lib.ifx_gemm_generic(a, w, bias, out, T, N, K, 0, 0, _stream()),
                   "gemm (float32)")
            self.launches += 1
            return out
        if T <= self.SKINNY_MAX_ROWS and K % 8 == 0 and a.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0:
            tiles = -(-N // 128)
            splits = self.skinny_slices(T, N, K) if allow_partial and bias is None else 1
            if splits > 1:
                parts = self.linear_skinny(a, w, None, splits=splits, mode=1, rows=rows)
                return PartialSum(parts, out_dtype)
            if tiles >= 74 or allow_partial or rows is not None:
                return self.linear_skinny(a, w, bias, out_dtype=out_dtype, splits=1, mode=0, rows=rows)
        out = torch.empty(T, N, dtype=out_dtype, device=a.device)
        _check(self.lib.ifx_gemm_cublas_bf16(a, w, out, T, N, K, _DT[out_dtype], _stream()),
               "gemm (bfloat16)")
        self.library_calls += 1
        if bias is not None:
            out += bias.to(out.dtype)
        return out

    @staticmethod
    def skinny_slices(rows, n, k):
        """Slices of K of a few-rows product whose consumer adds them.  Up to 128 rows: two blocks a SM and up to 10 slices;
        above, a block owns its SM (32 KB of activations a stage) and every slice costs a [rows, n] float32 round trip: at most 5."""
        slots, most = (296, 10) if rows <= 128 else (148, 5)
        return max(1, min(slots // -(-n // 128), most, -(-k // 64) // 4))

    def swiglu_few(self, a, w_gate_up, w_down):
        """A whole SwiGLU feed-forward of few bfloat16 rows, its two products launched by one call: what
        `linear(linear_swiglu(a, w_gate_up), w_down, allow_partial=True)` gives, or None where that does not take the
        few-rows kernels twice.  The host's time bounds such a call on small layers."""
        rows = a if isinstance(a, ScaledRows) else None
        if rows is not None:
            a = rows.pre
        T, K = a.shape
        N, inter = w_down.shape
        if not (a.dtype == w_gate_up.dtype == w_down.dtype == torch.bfloat16 and 0 < T <= self.SKINNY_MAX_ROWS and K % 8 == 0
                and inter % 8 == 0 and tuple(w_gate_up.shape) == (2 * inter, K) and a.is_contiguous() and w_gate_up.is_contiguous()
                and w_down.is_contiguous() and (a.data_ptr() | w_gate_up.data_ptr() | w_down.data_ptr()) % 16 == 0):
            return None
        splits = self.skinny_slices(T, N, inter)
        hidden = torch.empty(T, inter, dtype=torch.bfloat16, device=a.device)
        out = (torch.empty(splits, T, N, dtype=torch.float32, device=a.device) if splits > 1
               else torch.empty(T, N, dtype=torch.bfloat16, device=a.device))
        _check(self.lib.ifx_swiglu_few(a, w_gate_up, w_down, hidden, out, out, T, K, inter, N, splits,
                                       (None if rows is None else rows.sumsq), 0 if rows is None else rows.sumsq.shape[1],
                                       float(0.0 if rows is None else rows.eps), self.error_flag, _stream()),
               "swiglu (few rows)")
        self.launches += 2
        return PartialSum(out, torch.bfloat16) if splits > 1 else out

    @staticmethod
    def float32_by_parts(n, k):
        """Whether a float32 product runs on the tensor cores, its operands cut into three bfloat16 numbers each
        (csrc/gemm_f32_split.cu).  By the weight's sizes alone: a row's bits must not depend on how many there are.  Parts
        against the chain of multiply-adds, us, 1 / 16 / 100 / 512 rows: 1,536 x 1,368 24 25 27 41 against 29 25 45 81;
        2,048 x 1,024 18 17 21 34 against 17 17 29 70; 4,096 x 512 17 17 21 35 against 10 10 22 60; 1,024 x 1,024
        17 17 20 24 against 16 17 19 39; 256 x 8,192 20 24 29 41 against 97 99 123 123."""
        return k % 8 == 0 and k >= 1280 and n * k >= 1 << 21

    # The many-rows tcgen05 product with SiLU(gate)*up in its epilogue against cuBLAS followed by the activation
    # kernel, measured on a B200 (us a layer, 256 / 512 / 2,048 rows): Qwen2.5-1.5B sizes 18 vs 29, 25 vs 31, 77 vs 95;
    # 7B sizes 57 vs 79, 99 vs 106, 340 vs 382; 32B sizes (inner size 5,120) 111 vs 144, 197 vs 218, 767 vs 961; inner size
    # 8,192 (28,672 outputs) 208 vs 221, 347 vs 397, 1,297 vs 1,564.  The line comes from tiles of single SMs, which were
    # slower than the library's at 5,120 (851 vs 779 us at 2,048 rows); by pairs of SMs they are ahead there too.  It stays for
    # what it does to results: beyond it gate and up are rounded to bfloat16 in front of the activation.
    SWIGLU_TILES_MAX_K = 4096

    def linear_swiglu(self, a, w_gate_up):
        """silu(a . Wg^T) * (a . Wu^T) with Wg and Wu stacked in w_gate_up [2 I, K]: one kernel
        with both accumulators for few rows, else the product followed by the activation kernel."""
        rows = a if isinstance(a, ScaledRows) else None
        if rows is not None:
            a = rows.pre
        T, K = a.shape
        inter = w_gate_up.shape[0] // 2
        if (a.dtype == torch.bfloat16 and 0 < T <= self.SKINNY_MAX_ROWS and K % 8 == 0 and a.data_ptr() % 16 == 0
                and w_gate_up.data_ptr() % 16 == 0):
            return self.linear_skinny(a, w_gate_up, None, splits=1, mode=2, n_out=inter, up_row_offset=inter, rows=rows)
        if rows is not None:
            a = self.materialize_rows(rows)
        if (self.swiglu_tiles and a.dtype == torch.bfloat16 and K % 8 == 0 and K <= self.SWIGLU_TILES_MAX_K
                and a.data_ptr() % 16 == 0 and w_gate_up.data_ptr() % 16 == 0 and a.is_contiguous()):
            return self.linear_tiles(a, w_gate_up, swiglu=True)        # many rows: own tcgen05 tiles, activation fused
        return self.silu_mul(self.linear(a, w_gate_up))

    def linear_geglu(self, a, w_gate_up, bias):
        """gelu_tanh(a . Wg^T + bg) * (a . Wu^T + bu) with Wg and Wu stacked in w_gate_up [2 I, K] and the biases (float32, or
        None) likewise: the activation in the product's epilogue as in `linear_swiglu`, else the product followed by the
        activation kernel."""
        T, K = a.shape
        inter = w_gate_up.shape[0] // 2
        _need(a.dtype == w_gate_up.dtype and w_gate_up.shape[1] == K and a.is_contiguous() and w_gate_up.is_contiguous()
              and (bias is None or (bias.dtype == torch.float32 and bias.is_contiguous() and bias.numel() == 2 * inter)),
              "linear_geglu: bad operands")
        if (T and a.dtype == torch.bfloat16 and K % 8 == 0 and a.data_ptr() % 16 == 0 and w_gate_up.data_ptr() % 16 == 0):
            few = T <= self.SKINNY_MAX_ROWS
            if few or (self.swiglu_tiles and K <= self.SWIGLU_TILES_MAX_K):
                out = torch.empty(T, inter, dtype=torch.bfloat16, device=a.device)
                product = self.lib.ifx_gemm_skinny_geglu if few else self.lib.ifx_gemm_tcgen05_geglu
                _check(product(a, w_gate_up, bias, out, T, inter, K, self.error_flag, _stream()),
                       "linear_geglu")
                self.launches += 1
                return out
        both = self.linear(a, w_gate_up)
        out = torch.empty(T, inter, dtype=a.dtype, device=a.device)
        _check(self.lib.ifx_geglu_mul(both, bias, out, T, inter, _DT[a.dtype], _stream()), "geglu_mul")
        self.launches += 1
        return out

    def linear_xielu(self, a, w, a_pos, a_neg):
        """xielu(a . w^T): for few bfloat16 rows and a product wide enough to fill the SMs without K slices, the
        weight-streaming kernel with the activation on its result; otherwise the product (maybe in K slices)
        followed by the activation kernel, which adds the slices."""
        T, K = a.shape
        N = w.shape[0]
        if (a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and 0 < T <= self.SKINNY_MAX_ROWS and K % 8 == 0
                and a.is_contiguous() and w.is_contiguous() and w.shape[1] == K and a.data_ptr() % 16 == 0
                and w.data_ptr() % 16 == 0 and -(-N // 128) >= 74):
            out = torch.empty(T, N, dtype=torch.bfloat16, device=a.device)
            _check(self.lib.ifx_gemm_skinny_act(a, w, None, out, T, N, K, w.shape[0], 0, None, 0,
                                                0.0, 1, float(a_pos), float(a_neg),
                                                self.error_flag, _stream()), "gemm_skinny (xielu)")
            self.launches += 1
            return out
        return self.xielu(self.linear(a, w, allow_partial=True), a_pos, a_neg)

    def linear_relu2(self, a, w):
        """max(a . w^T, 0)^2: the activation on the product's result inside the weight-streaming kernel (few bfloat16 rows, a
        product wide enough without K slices) or the tcgen05 tiles (many), else by the kernel that adds the slices."""
        T, K = a.shape
        N = w.shape[0]
        if (T and a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and K % 8 == 0 and a.is_contiguous() and w.is_contiguous()
                and w.shape[1] == K and a.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0):
            out = None
            if T <= self.SKINNY_MAX_ROWS and -(-N // 128) >= 74:
                out = torch.empty(T, N, dtype=torch.bfloat16, device=a.device)
                _check(self.lib.ifx_gemm_skinny_act(a, w, None, out, T, N, K, N, 0, None, 0,
                                                    0.0, 3, 0.0, 0.0,
                                                    self.error_flag, _stream()), "gemm_skinny (relu2)")
            elif T > self.SKINNY_MAX_ROWS and self.swiglu_tiles and K <= self.SWIGLU_TILES_MAX_K:
                out = torch.empty(T, N, dtype=torch.bfloat16, device=a.device)
                _check(self.lib.ifx_gemm_tcgen05(a, w, out, T, N, K, N, 6, 0, self.error_flag, _stream()),
                       "gemm_tcgen05 (relu2)")
            if out is not None:
                self.launches += 1
                return out
        return self.relu2(self.linear(a, w, allow_partial=True))

    def relu2(self, z):
        """max(z, 0)^2, element by element, in z's dtype; a PartialSum's slices are added first, in the same pass."""
        splits, out_dtype = 1, z.dtype
        if isinstance(z, PartialSum):
            out_dtype, splits, z = z.dtype, z.splits, z.parts
        _need(z.is_contiguous(), "relu2: contiguous input")
        out = torch.empty(tuple(z.shape[-2:]), dtype=out_dtype, device=z.device)
        _check(self.lib.ifx_relu2(z, out, (out.numel()), _DT[z.dtype], _DT[out_dtype], splits,
                                  _stream()), "relu2")
        self.launches += 1
        return out

    def check_errors(self):
        """Raise if a kernel reported that one of its bounded waits ran out (reads the device flag)."""
        code = int(self.error_flag.item())
        if code:
            self.error_flag.zero_()
            raise KernelError(f"a kernel gave up waiting on a barrier (code {code}); its output is not valid")

    def linear_skinny(self, a, w, bias=None, out_dtype=None, splits=1, mode=0, n_out=None, up_row_offset=0, rows=None):
        """The tcgen05 weight-streaming product for up to 256 token rows.
        mode 0: out[T, N] (+bias); mode 1: float32 partial sums [splits, T, N]; mode 2: silu(gate) * up.
        `rows`: the ScaledRows whose `pre` is `a`; the product then applies their row scale."""
        T, K = a.shape
        N = n_out if n_out is not None else w.shape[0]
        _need(a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16, "linear_skinny: bfloat16 only")
        _need(a.is_contiguous() and w.is_contiguous() and w.shape[1] == K, "linear_skinny: bad operands")
        out_dtype = out_dtype or torch.bfloat16
        out = partials = None
        if mode == 1:
            partials = torch.empty(splits, T, N, dtype=torch.float32, device=a.device)
        else:
            out = torch.empty(T, N, dtype=out_dtype, device=a.device)
        _check(self.lib.ifx_gemm_skinny(a, w, bias, out, partials, T, N, K, w.shape[0],
                                        splits, mode, up_row_offset, int(out_dtype == torch.float32),
                                        (None if rows is None else rows.sumsq),
                                        0 if rows is None else rows.sumsq.shape[1],
                                        float(0.0 if rows is None else rows.eps),
                                        self.error_flag, _stream()), "gemm_skinny")
        self.launches += 1
        return partials if mode == 1 else out

    def linear_tiles(self, a, w, swiglu=False):
        """The many-rows tcgen05 product (csrc/gemm_tcgen05.cu): a . w^T in bfloat16, or, with `swiglu`,
        silu(a . Wg^T) * (a . Wu^T) for w = [Wg; Wu] stacked, without the [T, 2 I] round trip."""
        T, K = a.shape
        _need(a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16, "linear_tiles: bfloat16 only")
        _need(a.is_contiguous() and w.is_contiguous() and w.shape[1] == K and K % 8 == 0, "linear_tiles: bad operands")
        N = w.shape[0] // 2 if swiglu else w.shape[0]
        out = torch.empty(T, N, dtype=torch.bfloat16, device=a.device)
        _check(self.lib.ifx_gemm_tcgen05(a, w, out, T, N, K, w.shape[0], int(bool(swiglu)),
                                         N if swiglu else 0, self.error_flag, _stream()), "gemm_tcgen05")
        self.launches += 1
        return out

    def linear_generic(self, a, w, bias=None, out_dtype=None):
        """The CUDA-core product for any dtype (used by tests and as the refusal-free path)."""
        T, K = a.shape
        N = w.shape[0]
        out_dtype = out_dtype or a.dtype
        out = torch.empty(T, N, dtype=out_dtype, device=a.device)
        _check(self.lib.ifx_gemm_generic(a, w, bias, out, T, N, K, _DT[a.dtype],
                                         _DT[out_dtype], _stream()), "gemm_generic")
        self.launches += 1
        return out

    # ------------------------------------------------------------ whole layers
    def _native_parts(self, block):
        """The block's (mixer, ffn, norm before the mixer, norm before the ffn) if it is exactly the arrangement
        and the parts that csrc/layer_forward.cu runs (no subclass: one may have changed a forward), else None."""
        known = getattr(block, "_native_parts", False)
        if known is not False:
            return known
        from ..parts.attention import Attention
        from ..parts.block import PreNormBlock
        from ..parts.mlp import SwiGLU
        from ..parts.norm import RMSNorm
        parts = None
        if type(block) is PreNormBlock:
            m, f, n1, n2 = block.mixer, block.ffn, block.norm_mixer, block.norm_ffn
            if (type(m) is Attention and not m.general and type(f) is SwiGLU and type(n1) is RMSNorm and type(n2) is RMSNorm
                    and m.hidden == f.hidden == n1.size == n2.size):
                parts = (m, f, n1, n2)
        block._native_parts = parts
        block._native_layers = {}
        return parts

    def _native_workspace(self, T, parts):
        m, f = parts[0], parts[1]
        need = int(self.lib.ifx_layer_workspace_bytes(T, m.hidden, m.nq * m.d, m.nkv * m.d, f.inter, self.SKINNY_MAX_ROWS))
        ws = self._layer_ws
        if ws is None or ws.numel() < need:
            if torch.cuda.is_current_stream_capturing():
                return None                              # no allocation inside a graph: the parts run one by one
            # graphs captured earlier hold the old one's address: it stays alive
            ws = torch.empty(max(need, 2 * (0 if ws is None else ws.numel())), dtype=torch.uint8, device=self.device)
            self._layer_ws_all.append(ws)
            self._layer_ws = ws
            self._layer_views = {}
        return ws

    def _native_layer_args(self, block, parts, ctx, cache):
        """The C structure of one layer with one cache (sizes, constants, weight and cache addresses), made when
        the pair first runs and kept on the block; None if the cache or the weights are not bfloat16."""
        m, f, n1, n2 = parts
        tensors = (m.w_qkv, m.w_o, m.b_qkv, f.w_gate_up, f.w_down, n1.weight, n2.weight)
        kv, table = cache.kv, cache.block_table
        kv_ptr = kv.data_ptr()
        # everything of the cache that the structure holds: another runner may get the same addresses
        key = (kv_ptr, table.data_ptr(), cache.writes, cache.page_size, table.shape[1], kv.shape[0])
        entry = block._native_layers.get(key)
        if entry is None or any(a is not b for a, b in zip(entry[1], tensors)):
            if kv.dtype is not torch.bfloat16 or m.w_qkv.dtype is not torch.bfloat16:
                return None
            rotary = m.position.rotary(ctx.device) if m.position is not None else None
            la = _LayerArgs(
                hidden=m.hidden, inter=f.inter, nq=m.nq, nkv=m.nkv, d=m.d, window=int(m.window or 0),
                rot=0 if rotary is None else int(rotary.rotary_dim),
                interleaved=int(bool(rotary.interleaved)) if rotary is not None else 0,
                scale=m.scale, eps_in=n1.eps, eps_post=n2.eps, write_cache=int(bool(cache.writes)),
                norm_in_w=n1.weight.data_ptr(), norm_post_w=n2.weight.data_ptr(),
                b_qkv=0 if m.b_qkv is None else m.b_qkv.data_ptr(),
                inv_freq=0 if rotary is None else rotary.inv_freq.data_ptr(),
                w_qkv=m.w_qkv.data_ptr(), w_o=m.w_o.data_ptr(), w_gate_up=f.w_gate_up.data_ptr(),
                w_down=f.w_down.data_ptr(), kv_pool=kv_ptr, block_table=table.data_ptr(),
                max_blocks=table.shape[1], page_size=cache.page_size, num_pages=kv.shape[0])
            entry = (la, tensors, rotary, table, ctypes.byref(la))      # the tensors stay alive with the addresses
            if len(block._native_layers) >= 8:           # caches come and go with their runners
                block._native_layers.clear()
            block._native_layers[key] = entry
        return entry[4]

    def _native_step_args(self, ctx, device):
        """The C structure of the step's batch (metadata addresses, counts, this table's knobs), made at the
        step's first layer and kept on the context."""
        step = getattr(ctx, "_native_step", None)
        if step is None or step[1] is not ctx.positions or step[0].max_kv_len != ctx.max_kv_len:
            if "attn.prefill_tiles" not in ctx.extra:      # a step context built without the mixer as a provider
                for name, vals in self.attention_sections(ctx).items():
                    ctx.extra[name] = torch.tensor(vals, dtype=torch.int32, device=device)
                    ctx.extra_len[name] = len(vals)
            sa = _StepArgs(
                T=ctx.num_tokens, num_decode=ctx.extra_len["attn.decode_rows"],
                num_tiles=ctx.extra_len["attn.prefill_tiles"] // 4,
                max_kv_len=int(ctx.max_kv_len), positions=ctx.positions.data_ptr(), token_req=ctx.token_req.data_ptr(),
                req_slot=ctx.req_slot.data_ptr(), decode_rows=ctx.extra["attn.decode_rows"].data_ptr(),
                decode_meta=ctx.extra["attn.decode_meta"].data_ptr(),
                prefill_tiles=ctx.extra["attn.prefill_tiles"].data_ptr(), norm_sumsq=self._norm_sumsq.data_ptr(),
                norm_tickets=self._norm_tickets.data_ptr(), error_flag=self.error_flag.data_ptr(),
                skinny_max_rows=self.SKINNY_MAX_ROWS, swiglu_tiles=int(self.swiglu_tiles),
                swiglu_tiles_max_k=self.SWIGLU_TILES_MAX_K, tensor_core_prefill=int(self.tensor_core_prefill),
                overlap_attention=int(self.overlap_attention))
            step = ctx._native_step = (sa, ctx.positions, ctypes.byref(sa))
        return step[2]

    def fused_prenorm_layer(self, block, x, pending, ctx, cache):
        """One native call for a pre-norm layer of attention and SwiGLU in bfloat16: the kernels that the parts
        would launch one by one, chosen by the same rules, launched from csrc/layer_forward.cu.  Returns
        (x, the layer's last delta, unadded) or None if this block, dtype or cache is not what that code runs."""
        if not self.native_layers or ctx.dtype is not torch.bfloat16 or cache.kv is None or cache.block_table is None:
            return None
        parts = self._native_parts(block)
        if parts is None or x.dtype is not torch.float32:
            return None
        m, f, n1, n2 = parts
        if block.mixer is not m or block.ffn is not f or block.norm_mixer is not n1 or block.norm_ffn is not n2:
            block._native_parts = False                  # a part was exchanged: look again
            return self.fused_prenorm_layer(block, x, pending, ctx, cache)
        T = ctx.num_tokens
        ws = self._native_workspace(T, parts)
        if ws is None:
            return None
        layer = self._native_layer_args(block, parts, ctx, cache)
        if layer is None:
            return None
        step = self._native_step_args(ctx, x.device)
        io = self._layer_io
        io.x = x.data_ptr()
        if pending is None:
            io.pending_tensor, io.pending_parts, io.pending_splits = 0, 0, 0
        elif isinstance(pending, PartialSum):
            if tuple(pending.shape) != tuple(x.shape):
                return None
            io.pending_tensor, io.pending_parts, io.pending_splits = 0, pending.parts.data_ptr(), pending.splits
        else:
            if pending.dtype is not torch.bfloat16 or pending.shape != x.shape or not pending.is_contiguous():
                return None
            io.pending_tensor, io.pending_parts, io.pending_splits = pending.data_ptr(), 0, 0
        parity = self._layer_parity = 1 - self._layer_parity
        io.parity = parity
        io.least_decode_splits = self.least_decode_splits(ctx, ctx.extra_len.get("attn.decode_rows", 0), m.nkv, m.d, int(m.window or 0))
        io.prefill_parts = self.prefill_cut(ctx, m.nq, int(m.window or 0))
        io.ws, io.ws_bytes = ws.data_ptr(), ws.numel()
        rc = self.lib.ifx_layer_forward(step, layer, self._layer_io_ref, ctypes.c_void_p(_stream()))
        self.launches += io.launches
        self.library_calls += io.library_calls
        self.native_layer_calls += 1
        _check(rc, "layer (native)")
        view = (T, m.hidden, parity, io.out_splits)
        out = self._layer_views.get(view)
        if out is None:
            at = (io.out_parts or io.out_tensor) - ws.data_ptr()
            if io.out_splits:
                n = io.out_splits * T * m.hidden * 4
                out = PartialSum(ws[at:at + n].view(torch.float32).view(io.out_splits, T, m.hidden), torch.bfloat16)
            else:
                out = ws[at:at + T * m.hidden * 2].view(torch.bfloat16).view(T, m.hidden)
            self._layer_views[view] = out
        return x, out

    # --------------------------------------------------------------- attention
    PREFILL_TILE = 256         # query rows per work item of the prompt-portion attention kernels

    def attention_sections(self, ctx):
        """Work lists of the attention kernels for one step, from the step's spans:
        attn.decode_rows[D] (flat indices of spans of one token), attn.decode_meta[D,4] (flat index,
        position, slot, 0: what the decode kernel needs of a token, in one 16-byte load),
        attn.prefill_tiles[P,4] (request, first flat row, rows, first position) for longer spans."""
        rows, single, tiles, base = [], [], [], 0
        for r, ((start, n), slot) in enumerate(zip(ctx.spans, ctx.slots_host)):
            if n == 1:
                rows.append(base)
                single.append((base, start, int(slot), 0))
            else:
                for off in range(0, n, self.PREFILL_TILE):
                    tiles.extend((r, base + off, min(self.PREFILL_TILE, n - off), start + off))
            base += n
        # Longest first, for then no long one starts when the others end (28 heads, 40 tokens at up to 4,200 keys: 62.0 -> 56.4 us;
        # 64 at up to 8,000: 108 -> 105).  Up to 16 tokens all blocks run at once whatever the order (8 tokens: 22.4, sorted 23.6).
        if len(single) > 16:
            single.sort(key=lambda m: -m[1])
        # (longest, sum) of the decoded tokens' keys, for least_decode_splits; a captured step takes it back
        ctx.__dict__.pop("prefill_parts", None)            # what an earlier list of spans gave
        ctx.decode_keys = (1 + max(m[1] for m in single), len(single) + sum(m[1] for m in single)) if single else None
        return {"attn.decode_rows": rows, "attn.decode_meta": [v for m in single for v in m], "attn.prefill_tiles": tiles}

    @staticmethod
    def small_attention_grid(ctx, nkv):
        """1 if the step is decoded tokens only and their attention grid (tokens x kv heads x up to 8 key slices)
        leaves SMs free: the rotation kernel then lets it in early."""
        extra_len = getattr(ctx, "extra_len", None) or {}
        if "attn.decode_rows" not in extra_len:
            return 0
        return int(extra_len.get("attn.prefill_tiles", 0) == 0 and extra_len["attn.decode_rows"] * nkv * 8 <= 148)

    def rope_append(self, qkv, bias, rotary, nq, nkv, d, ctx, cache, q_norm=None, k_norm=None, norm_eps=0.0, dv=None,
                    own_kv=True, q_temp=None):
        """`qkv`: the stacked projections [T, (nq + 2 nkv) d] as a tensor or a PartialSum.
        With `q_norm` / `k_norm` (float32 [d]) every query / key head is RMS-normed with that weight before the
        rotation; `dv`: the values' head size if it is not `d` (cache rows hold the larger of the two);
        `own_kv` False: the rows hold queries only and nothing is stored; `q_temp` = (coef, every): the queries are
        multiplied by 1 + coef ln(floor((p + 1) / every) + 1) at position p.  A table whose cos and sin are made longer
        (`rotary.magnitude`) or cache rows longer than a head take the general kernel too."""
        if (q_norm is not None or k_norm is not None or (dv is not None and dv != d) or not own_kv or q_temp is not None
                or (rotary is not None and rotary.magnitude != 1.0) or (cache.kv is not None and cache.kv.shape[-1] != d)):
            return self._norm_rope_append(qkv, bias, rotary, nq, nkv, d, ctx, cache, q_norm, k_norm, norm_eps,
                                          d if dv is None else dv, own_kv, q_temp)
        partial, splits = None, 0
        if isinstance(qkv, PartialSum):
            partial, splits, dtype, device = qkv.parts, qkv.splits, qkv.dtype, qkv.parts.device
            T, width = qkv.shape
            qkv = None
        else:
            dtype, device = qkv.dtype, qkv.device
            T, width = qkv.shape
        _need(width == (nq + 2 * nkv) * d, "rope_append: qkv width does not fit the head counts")
        q_out = torch.empty(T, nq * d, dtype=dtype, device=device)
        write = bool(cache.writes and cache.kv is not None)
        kv, table = cache.kv, cache.block_table
        if write:
            if kv.dtype != dtype:
                raise KernelError(f"rope_append: cache is {kv.dtype}, activations {dtype}")
        rot = 0 if rotary is None else int(rotary.rotary_dim)
        _need(rot <= d, "rope_append: rotary_dim exceeds the head size")
        _check(self.lib.ifx_rope_append(
            qkv, partial, splits, bias, (None if rotary is None else rotary.inv_freq), rot,
            int(bool(rotary.interleaved)) if rotary is not None else 0,
            ctx.positions, ctx.token_req, ctx.req_slot, table,
            0 if table is None else table.shape[1], cache.page_size, 0 if kv is None else kv.shape[0],
            kv, q_out, T, nq, nkv, d, int(write), self.small_attention_grid(ctx, nkv), _DT[dtype],
            _stream()), "rope_append")
        self.launches += 1
        return q_out

    def _norm_rope_append(self, qkv, bias, rotary, nq, nkv, d, ctx, cache, q_norm, k_norm, norm_eps, dv, own_kv, q_temp=None):
        _need(bias is None, "rope_append: biases and head norms together are not built")
        partial, splits = None, 0
        if isinstance(qkv, PartialSum):
            partial, splits, dtype, device = qkv.parts, qkv.splits, qkv.dtype, qkv.parts.device
            T, width = qkv.shape
            qkv = None
        else:
            dtype, device = qkv.dtype, qkv.device
            T, width = qkv.shape
        src_kv = nkv if own_kv else 0
        _need(width == (nq + src_kv) * d + src_kv * dv, "rope_append: the rows' width does not fit the head counts")
        for w in (q_norm, k_norm):
            _need(w is None or (w.dtype == torch.float32 and w.numel() == d), "rope_append: a head norm weight is float32 [d]")
        q_out = torch.empty(T, nq * d, dtype=dtype, device=device)
        kv, table = cache.kv, cache.block_table
        write = bool(own_kv and cache.writes and kv is not None)
        d_row = d
        if write:
            if kv.dtype != dtype:
                raise KernelError(f"rope_append: cache is {kv.dtype}, activations {dtype}")
            d_row = kv.shape[-1]
            _need(kv.shape[1] == 2 and kv.shape[2] == nkv and d_row >= max(d, dv), "rope_append: the cache does not fit the heads")
        rot = 0 if rotary is None else int(rotary.rotary_dim)
        _need(rot <= d, "rope_append: rotary_dim exceeds the head size")
        _check(self.lib.ifx_norm_rope_append_ex(
            qkv, partial, splits, q_norm, k_norm, float(norm_eps),
            (None if rotary is None else rotary.inv_freq), rot,
            int(bool(rotary.interleaved)) if rotary is not None else 0, ctx.positions, ctx.token_req,
            ctx.req_slot, table, 0 if table is None else table.shape[1], cache.page_size,
            0 if kv is None else kv.shape[0], (kv if write else None), q_out, T, nq, src_kv, nkv, d, dv, d_row,
            int(write), float(1.0 if rotary is None else rotary.magnitude),
            float(0.0 if q_temp is None else q_temp[0]), 0 if q_temp is None else int(q_temp[1]),
            _DT[dtype], _stream()), "rope_append (normed heads)")
        self.launches += 1
        return q_out

    def attention(self, q, nq, nkv, d, window, scale, ctx, cache, chunk=None, sink=False, dv=None, turn_back=None,
                  keep_first=0, head_gate=None):
        """Every token attends its request's keys up to its own position (or the last
        `window` of them) through the block table.  float32: the per-token kernel
        whose additions depend on the position only.  bfloat16: the tiled kernels,
        one launch for the prompt portions and one for the single decoded tokens.
        `chunk`: a query at position p sees keys from (p // chunk) * chunk on; `sink`: one more unit in the
        softmax's denominator (True), or exp of a learned number per head (a float32 tensor [nq]); `dv`: the values'
        head size if it is not `d`; `turn_back`: what `row_norm_rope_append` returned for values that were turned, so that
        every head's output is turned back by the query's position before it is rounded; `keep_first`: the first keys of a
        sequence that every query sees besides its window or chunk; `head_gate` (float32 [T, nq]): every head's output is
        multiplied by it before it is rounded."""
        if (turn_back is not None or keep_first or head_gate is not None or chunk or torch.is_tensor(sink) or sink or (dv is not None and dv != d)
                or (cache.kv is not None and cache.kv.shape[-1] != d)):      # cache rows longer than a head
            return self._attention_masked(q, nq, nkv, d, d if dv is None else dv, window, chunk, sink, scale, ctx, cache,
                                          turn_back, int(keep_first), head_gate)
        T = q.shape[0]
        kv, table = cache.kv, cache.block_table
        _need(kv is not None and table is not None, "attention: the mixer has no key/value cache")
        if kv.dtype != q.dtype:
            raise KernelError(f"attention: cache is {kv.dtype}, queries {q.dtype}")
        if d % 8 or d > 256:
            raise KernelError(f"attention: head size {d} is not a multiple of 8 up to 256")
        _need(q.is_contiguous() and q.shape[1] == nq * d, "attention: queries must be one [tokens, heads * size] block")
        out = torch.empty(T, nq * d, dtype=q.dtype, device=q.device)
        win = 0 if window is None else int(window)
        common = (cache.page_size, table.shape[1], kv.shape[0], win, float(scale))
        tiled = q.dtype == torch.bfloat16 and bool(self.lib.ifx_attention_mma_supports(d))
        if "attn.prefill_tiles" not in ctx.extra:          # a step context built without the mixer as a provider
            for name, vals in self.attention_sections(ctx).items():
                ctx.extra[name] = torch.tensor(vals, dtype=torch.int32, device=q.device)
                ctx.extra_len[name] = len(vals)
        tiles, num_tiles = ctx.extra["attn.prefill_tiles"], ctx.extra_len["attn.prefill_tiles"] // 4
        decode_rows, decode_meta = ctx.extra["attn.decode_rows"], ctx.extra["attn.decode_meta"]
        if not tiled:
            self._attention_generic(q, kv, table, ctx, None, T, out, nq, nkv, d, common)
            return out
        if num_tiles and self.tensor_core_prefill and self.lib.ifx_attention_prefill_tcgen05_supports(
                d, cache.page_size):
            parts = self.prefill_cut(ctx, nq, win)
            room = None
            if parts > 1:
                room = torch.empty(self.prefill_parts_bytes(num_tiles, nq, d, parts), dtype=torch.uint8, device=q.device)
                self.launches += 1
            _check(self.lib.ifx_attention_prefill_tcgen05_parts(
                q, T, kv, table, tiles, ctx.req_slot, out,
                num_tiles, nq, nkv, d, *common, parts, room, self.error_flag, _stream()),
                "attention (prompt portions, tcgen05)")
            self.launches += 1
        elif num_tiles:
            _check(self.lib.ifx_attention_prefill_bf16(
                q, kv, table, tiles, ctx.req_slot, out,
                num_tiles, nq, nkv, d, *common, int(ctx.max_kv_len), self.error_flag, _stream()),
                "attention (prompt portions)")
            self.launches += 1
        n = ctx.extra_len["attn.decode_rows"]
        if n:
            if nq // nkv > 16:
                self._attention_generic(q, kv, table, ctx, decode_rows, n, out, nq, nkv, d, common)
                return out
            max_keys = int(ctx.max_kv_len if not win else min(win, ctx.max_kv_len))
            most = int(self.lib.ifx_attention_decode_max_splits(d, cache.page_size))
            splits = max(self.decode_splits(n, nkv, max_keys, most), min(most, self.least_decode_splits(ctx, n, nkv, d, win)))
            _check(self.lib.ifx_attention_decode_bf16(
                q, kv, table, decode_meta, out, n, nq, nkv, d, *common, splits,
                max_keys, self.error_flag, _stream()), "attention (decoded tokens)")
            self.launches += 1
        return out

    PREFILL_PART_TILES = 4     # key tiles (of 128) that a part of a prompt attention block keeps at least

    @staticmethod
    def prefill_parts_bytes(num_tiles, nq, d, parts):
        """What ifx_attention_prefill_tcgen05_parts_bytes says: a sum of d numbers, a reference and a denominator per row of a part."""
        return num_tiles * nq % 148 * parts * 256 * (d + 2) * 4

    def prefill_parts(self, ctx, nq, window):
        """Parts of their keys that the prompt attention's left over blocks are cut into (1: whole), found once a step and kind of layer."""
        known = ctx.__dict__.setdefault("prefill_parts", {})
        parts = known.get((nq, window))
        if parts is None:
            parts = known[nq, window] = self._prefill_parts(ctx, nq, window)
        return parts

    def prefill_cut(self, ctx, nq, window):
        """What the kernel is told: prefill_parts, or -1 for a block for each 128 rows; found once a step and kind of layer."""
        known = ctx.__dict__.setdefault("prefill_parts", {})
        cut = known.get((nq, window, "cut"))
        if cut is None:
            cut = self.prefill_parts(ctx, nq, window)
            if cut == 1 and self._prefill_by_tiles(ctx, nq):
                cut = -1
            known[nq, window, "cut"] = cut
        return cut

    @staticmethod
    def _prefill_by_tiles(ctx, nq):
        """Whether each 128 rows get a block of their own instead of 256 rows: while all of those fit on the SMs at once, and the block that
        walks the most keys is one of two query tiles.  Such a block takes an eighth longer a key tile, and the second tile's last keys
        and its output come behind the first one's, two thirds of a key tile.  Where a block of one query tile walks longer, nothing is
        gained, and the second query tiles that are not there, which are launched all the same and leave at once, cost up to 4 us.
        us, 256 and 128 rows a block: 12 heads, 447 tokens 13.3 and 11.8, 1,000 20.0 and 18.2, with four of 50 beside 20.0 and 18.4, four
        times 256 behind 700 20.7 and 18.7; 28 heads, 300 behind 500 17.4 and 17.1, 640 behind 1,500 35.1 and 32.8; heads of 64, 16 of
        them, 1,000 tokens 19.2 and 15.9; and those that stay: 12 heads, 300 tokens 10.2 and 10.2, four times 300 10.8 and 12.0, twelve times
        100 8.6 and 11.8, behind 700 17.4 and 21.3.  With more blocks than SMs: 1,000 of 28 heads behind 2,000 48.4 and 68.6, 3,500 of 12
        55.0 and 65.0 (the last blocks of 2,000 of 12 alone are long enough to gain, 33.9 and 31.0, and are left)."""
        tiles = two = one = 0                              # 128-row tiles; keys to the end of the longest item of two tiles, and of one
        for s, n in ctx.spans:
            if n > 1:
                tiles += -(-n // 128)
                rest = n % 256
                if 0 < rest <= 128:
                    one = max(one, s + n)
                    n -= rest
                if n:
                    two = max(two, s + n)
        return tiles * nq <= 148 and two > 0 and 1.12 * -(-two // 128) + 0.7 > -(-one // 128)

    def _prefill_parts(self, ctx, nq, window):
        """A block takes up to 256 tokens of a head and an SM to itself, so what is left behind whole rounds of 148 blocks leaves SMs idle
        for as long as its longest block walks; with few blocks that is the whole grid.  Cut while every part keeps four tiles of 128
        keys: with parts of three or of six the times below are the same or up to 3 % longer, and below that adding the parts up takes
        what they save.  Eight tiles stay whole too: two parts of four save 0.6 us, and the launch that adds them up and its workspace
        cost the host 5.
        us, whole and cut: 28 heads, two requests' 2,500 tokens behind up to 4,000 (12 of 308 blocks left) 191 and 162, 384 tokens
        behind 2,000 39.0 and 32.4; 12 heads, 512 tokens behind 3,000 (24 blocks, six parts) 61.9 and 30.2, 600 tokens behind 900
        26.9 and 24.6."""
        blocks = ctx.extra_len["attn.prefill_tiles"] // 4 * nq
        left = blocks % 148
        if not 0 < left <= 74:
            return 1
        items, longest = -(-left // nq), 0                 # the first items' blocks run last
        for start, n in ctx.spans:
            if n == 1:
                continue
            for off in range(0, n, self.PREFILL_TILE):
                first, end = start + off, start + min(n, off + self.PREFILL_TILE)
                longest = max(longest, -(-end // 128) - (max(0, first - window + 1) // 128 if window else 0))
                items -= 1
                if not items:
                    return max(1, min(148 // left, longest // self.PREFILL_PART_TILES, 8)) if longest > 2 * self.PREFILL_PART_TILES else 1
        return 1

    @staticmethod
    def least_decode_splits(ctx, num_tokens, nkv, d, window):
        """Parts that a decoded token's keys are cut into at least, where the tokens of a step have uneven numbers of keys: with a
        block a token and head the longest alone decides how long the step takes, and the others' SMs idle.  Parts cost a
        prologue and a merge each, so a token's keys have to be long, and even steps, whose blocks end together, keep
        decode_splits.  us, heads of 128, with 1 / 2 / 4 parts, longest first: 28 + 4 heads, 40 tokens at 4,400 keys in the
        mean and 7,800 at most 87 / 65 / 62, 48 at 4,100 and 7,900 97 / 75 / 70, 64 at 4,400 and 7,900 105 / 102 / 97, 48 at 2,200 and
        4,100 63 / 56 / 58, 64 at 1,700 and 3,000 53.8 / 55.5 / 61; even, 64 at 4,096 82 / 90 / 100, 40 at 7,900 102 / 136 / 117;
        12 + 2 heads, 40 at 4,400 and 7,800 64 / 54 / 46, 48 at 2,900 and 5,800 51 / 46 / 40."""
        keys = getattr(ctx, "decode_keys", None)
        if keys is None or window or num_tokens * nkv > 296 or keys[0] * num_tokens * 2 < keys[1] * 3:
            return 1
        size = keys[0] * d
        return 4 if size >= 5600 * 128 else 2 if size >= 4000 * 128 else 1

    @staticmethod
    def decode_splits(num_tokens, nkv, max_keys, max_splits=8):
        """Into how many thread blocks (one cluster: 1, 2, 4, 8, or 16 where the kernel takes it) the
        key range of a decoded token is cut: as many blocks as the 148 SMs hold at once (two each), but
        at least 128 keys per block.  Clusters of 16 only while all of them fit on the SMs at once (measured:
        8.3 against 11.0 us for one token of the 7B shape at 4,096 keys, but 20 against 14 us for 16 clusters)."""
        want = max(1, 296 // max(1, num_tokens * nkv))           # all blocks resident at once: two a SM
        limit = max(1, min(want, max_keys // 128, max_splits))
        splits = 1
        while splits * 2 <= limit:
            splits *= 2
        if splits > 8 and num_tokens * nkv * splits > 148:
            splits = 8
        return splits

    def _attention_masked(self, q, nq, nkv, d, dv, window, chunk, sink, scale, ctx, cache, turn_back=None, keep_first=0,
                          head_gate=None):
        """Attention with a chunk mask, kept first keys, a sink, values of their own size, turned values or gated heads: the
        tiled kernels where they take the sizes, else the per-token kernel."""
        T = q.shape[0]
        kv, table = cache.kv, cache.block_table
        _need(kv is not None and table is not None, "attention: the mixer has no key/value cache")
        if kv.dtype != q.dtype:
            raise KernelError(f"attention: cache is {kv.dtype}, queries {q.dtype}")
        _need(q.is_contiguous() and q.shape[1] == nq * d, "attention: queries must be one [tokens, heads * size] block")
        d_row = kv.shape[-1]
        _need(kv.shape[1] == 2 and kv.shape[2] == nkv and d_row >= max(d, dv) and d_row % 8 == 0 and d_row <= 256,
              "attention: the cache does not fit the heads")
        out = torch.empty(T, nq * dv, dtype=q.dtype, device=q.device)
        win = 0 if window is None else int(window)
        sink_values = sink if torch.is_tensor(sink) else None
        if sink_values is not None:
            _need(sink_values.dtype == torch.float32 and sink_values.numel() == nq and sink_values.is_contiguous(),
                  "attention: the learned sink is float32 [heads]")
        back, neighbours = (None, 0) if turn_back is None else (turn_back[0], int(bool(turn_back[1])))
        _need(back is None or (back.dtype == torch.float32 and back.is_contiguous() and tuple(back.shape) == (T, dv // 2, 2)),
              "attention: cos and sin of the values' angles are float32 [tokens, dv / 2, 2]")
        _need(head_gate is None or (head_gate.dtype == torch.float32 and head_gate.is_contiguous()
                                    and tuple(head_gate.shape) == (T, nq)), "attention: a gate per head is float32 [tokens, heads]")
        if (q.dtype == torch.bfloat16 and d == dv == d_row and nq // nkv <= 16 and self.lib.ifx_attention_mma_supports(d)
                and os.environ.get("INFERFLUX_B200_MASKED_TILES", "1") != "0"):
            # the tiled kernels: prompt portions on mma.sync tiles, single tokens on the cluster kernel
            if "attn.prefill_tiles" not in ctx.extra:          # a step context built without the mixer as a provider
                for name, vals in self.attention_sections(ctx).items():
                    ctx.extra[name] = torch.tensor(vals, dtype=torch.int32, device=q.device)
                    ctx.extra_len[name] = len(vals)
            num_tiles = ctx.extra_len["attn.prefill_tiles"] // 4
            common = (cache.page_size, table.shape[1], kv.shape[0], win, int(chunk or 0),
                      int(sink_values is not None or bool(sink)), sink_values, float(scale), back, neighbours,
                      keep_first, head_gate)
            if num_tiles and self.tensor_core_prefill and self.lib.ifx_attention_prefill_tcgen05_supports(d, cache.page_size):
                _check(self.lib.ifx_attention_prefill_tcgen05_sink(
                    q, T, kv, table, ctx.extra["attn.prefill_tiles"], ctx.req_slot, out,
                    num_tiles, nq, nkv, d, *common, self.error_flag, _stream()),
                    "attention (masked, prompt portions, tcgen05)")
                self.launches += 1
            elif num_tiles:
                _check(self.lib.ifx_attention_prefill_bf16_sink(
                    q, kv, table, ctx.extra["attn.prefill_tiles"], ctx.req_slot, out,
                    num_tiles, nq, nkv, d, *common, int(ctx.max_kv_len), self.error_flag, _stream()),
                    "attention (masked, prompt portions)")
                self.launches += 1
            n = ctx.extra_len["attn.decode_rows"]
            if n:
                max_keys = int(ctx.max_kv_len)
                if win:
                    max_keys = min(max_keys, win)
                if chunk:
                    max_keys = min(max_keys, int(chunk))
                if keep_first:                              # (both ends in whole tiles of 16)
                    max_keys = min(int(ctx.max_kv_len), max_keys + -(-keep_first // 16) * 16)
                splits = self.decode_splits(n, nkv, max_keys, int(self.lib.ifx_attention_decode_max_splits(d, cache.page_size)))
                _check(self.lib.ifx_attention_decode_bf16_sink(
                    q, kv, table, ctx.extra["attn.decode_meta"], out, n, nq, nkv, d, *common,
                    splits, max_keys, self.error_flag, _stream()), "attention (masked, decoded tokens)")
                self.launches += 1
            return out
        _check(self.lib.ifx_attention_generic_sink(
            q, kv, table, ctx.positions, ctx.token_req, ctx.req_slot, None,
            out, T, nq, nkv, d, dv, d_row, cache.page_size, table.shape[1], kv.shape[0],
            0 if window is None else int(window), int(chunk or 0), int(sink_values is not None or bool(sink)),
            sink_values, float(scale), back, neighbours, keep_first, head_gate,
            _DT[q.dtype], _stream()), "attention (masked)")
        self.launches += 1
        return out

    def _attention_generic(self, q, kv, table, ctx, rows, count, out, nq, nkv, d, common):
        _check(self.lib.ifx_attention_generic(
            q, kv, table, ctx.positions, ctx.token_req, ctx.req_slot,
            rows, out, count, nq, nkv, d, *common, _DT[q.dtype], _stream()), "attention")
        self.launches += 1

    # ------------------------------------------- layers that norm a sublayer's output
    def postnorm_add(self, x, y, w_post, eps_post, w_next=None, eps_next=0.0, out_dtype=None, conv=None, cast_out=False,
                     groups=1, both=False):
        """x += y / rms(y) * w_post (x float32, in place).  With `w_next`, also returns the next norm of the
        updated rows, x / rms(x) * w_next in `out_dtype`: sum and both norms in one kernel.  With `cast_out`
        (and no `w_next`) it returns the updated rows themselves in `out_dtype`, for a sublayer that reads
        x without a norm.  `conv` =
        (weight [hidden, taps], taps, state, index, ctx), allowed when every request of the step brings one token
        (`ctx.max_span == 1`): the rows come back as h + conv(h) over time, and the state has moved on.
        `groups`: the next norm's root mean square is taken per group of the row.  `both` (with `conv`): returns
        (h, h + conv(h))."""
        if groups > 1 or both:
            return self._postnorm_add_groups(x, y, w_post, eps_post, w_next, eps_next, out_dtype, conv, groups, both)
        splits = 1
        if isinstance(y, PartialSum):                      # the slices are added in the same pass
            _need(tuple(y.shape) == tuple(x.shape), "postnorm_add: partial sums do not match x")
            out_dtype = out_dtype or y.dtype
            y, splits = y.parts, y.splits
        _need(x.dtype == torch.float32 and x.is_contiguous() and y.is_contiguous() and tuple(y.shape[-2:]) == tuple(x.shape),
              "postnorm_add: x must be float32 and y of its shape")
        _need(w_post.dtype == torch.float32 and (w_next is None or w_next.dtype == torch.float32),
              "postnorm_add: norm weights must be float32")
        T, H = x.shape
        out = None if (w_next is None and not cast_out) else torch.empty(T, H, dtype=out_dtype or y.dtype, device=x.device)
        cw, taps, st_ptr, stride, treq, rslot = None, 0, 0, 0, None, None
        if conv is not None:
            cw, taps, state, index, ctx = conv
            _need(w_next is not None and ctx.max_span == 1 and tuple(cw.shape) == (H, taps) and cw.dtype == torch.float32,
                  "postnorm_add: the convolution is fused only into steps of single tokens")
            if taps > 1:
                _need(state is not None and state.dtype == torch.float32 and state.is_contiguous()
                      and tuple(state.shape[2:]) == (taps - 1, H) and 0 <= index < state.shape[1],
                      "postnorm_add: the state does not fit the convolution")
                stride = state.shape[1] * (taps - 1) * H
                st_ptr = state.data_ptr() + 4 * index * (taps - 1) * H
            treq, rslot = ctx.token_req, ctx.req_slot
        _check(self.lib.ifx_postnorm_add_rmsnorm(
            x, y, w_post, float(eps_post), w_next, float(eps_next), out,
            T, H, _DT[y.dtype], _DT[(out_dtype or y.dtype)], splits, cw, taps, st_ptr, stride,
            treq, rslot, _stream()), "postnorm_add")
        self.launches += 1
        return out

    def _postnorm_add_groups(self, x, y, w_post, eps_post, w_next, eps_next, out_dtype, conv, groups, both):
        splits = 1
        if isinstance(y, PartialSum):
            _need(tuple(y.shape) == tuple(x.shape), "postnorm_add: partial sums do not match x")
            out_dtype = out_dtype or y.dtype
            y, splits = y.parts, y.splits
        _need(x.dtype == torch.float32 and x.is_contiguous() and y.is_contiguous() and tuple(y.shape[-2:]) == tuple(x.shape),
              "postnorm_add: x must be float32 and y of its shape")
        _need(w_next is not None and w_post.dtype == torch.float32 and w_next.dtype == torch.float32,
              "postnorm_add: a norm over groups needs both float32 norm weights")
        T, H = x.shape
        out_dtype = out_dtype or y.dtype
        out = torch.empty(T, H, dtype=out_dtype, device=x.device)
        out2, cw, taps, st_ptr, stride, treq, rslot = None, None, 0, 0, 0, None, None
        if conv is not None:
            cw, taps, state, index, ctx = conv
            _need(ctx.max_span == 1 and tuple(cw.shape) == (H, taps) and cw.dtype == torch.float32,
                  "postnorm_add: the convolution is fused only into steps of single tokens")
            if taps > 1:
                _need(state is not None and state.dtype == torch.float32 and tuple(state.shape[2:]) == (taps - 1, H)
                      and state.stride(3) == 1 and state.stride(2) == H and 0 <= index < state.shape[1],
                      "postnorm_add: the state does not fit the convolution")
                stride = state.stride(0)
                st_ptr = state.data_ptr() + 4 * index * state.stride(1)
            treq, rslot = ctx.token_req, ctx.req_slot
            out2 = torch.empty(T, H, dtype=out_dtype, device=x.device)
        _check(self.lib.ifx_groupnorm_stream(
            x, y, w_post, float(eps_post), w_next, float(eps_next), int(groups),
            out, out2, T, H, _DT[y.dtype], _DT[out_dtype], splits, cw, taps, st_ptr,
            stride, treq, rslot, _stream()), "postnorm_add (groups)")
        self.launches += 1
        if conv is None:
            return out
        return (out, out2) if both else out2

    def residual_add_scaled(self, x, a, b, scale, out_dtype=None):
        """x += scale * (a + b) (x float32, in place; b may be None; a and b tensors of x's shape or PartialSums).  With
        `out_dtype` also returns the updated rows in that dtype."""
        T, H = x.shape
        _need(x.dtype == torch.float32 and x.is_contiguous(), "residual_add_scaled: x must be contiguous float32")

        def operand(v):
            if v is None:
                return None, 0, 1
            if isinstance(v, PartialSum):
                _need(tuple(v.shape) == (T, H), "residual_add_scaled: partial sums do not match x")
                return v.parts, 0, v.splits
            _need(tuple(v.shape) == (T, H) and v.is_contiguous(), "residual_add_scaled: an operand does not match x")
            return v, _DT[v.dtype], 1
        pa, da, sa = operand(a)
        pb, db, sb = operand(b)
        out = None if out_dtype is None else torch.empty(T, H, dtype=out_dtype, device=x.device)
        _check(self.lib.ifx_residual_add_scaled(x, pa, da, sa, pb, db, sb, float(scale), out,
                                                0 if out is None else _DT[out_dtype], T, H, _stream()), "residual_add_scaled")
        self.launches += 1
        return out

    def scale_(self, values, factor):
        """values *= factor, in place (float32)."""
        _need(values.dtype == torch.float32 and values.is_contiguous(), "scale_: contiguous float32 values")
        _check(self.lib.ifx_scale_f32(values, (values.numel()), float(factor), _stream()), "scale_")
        self.launches += 1

    def gelu_mul_table(self, z, table, token_ids, first_column):
        """gelu_tanh(z) * table[token, first_column : first_column + z.shape[1]], in z's dtype."""
        T, dim = z.shape
        _need(z.is_contiguous() and table.is_contiguous() and table.dtype == z.dtype and token_ids.numel() == T
              and first_column + dim <= table.shape[1], "gelu_mul_table: rows and table of one dtype, columns inside the table")
        out = torch.empty_like(z)
        _check(self.lib.ifx_gelu_mul_table(z, table, token_ids, table.shape[1], int(first_column),
                                           table.shape[0], out, T, dim, _DT[z.dtype], _stream()), "gelu_mul_table")
        self.launches += 1
        return out

    def rmsnorm_columns(self, rows, col0, n, w, eps):
        """Columns col0 .. col0 + n of `rows`, RMS-normed with weight `w` (float32), as a tensor of their own."""
        T, ld = rows.shape
        _need(rows.is_contiguous() and w.dtype == torch.float32 and w.numel() == n and col0 + n <= ld,
              "rmsnorm_columns: the columns must lie inside contiguous rows")
        out = torch.empty(T, n, dtype=rows.dtype, device=rows.device)
        _check(self.lib.ifx_latent_norm_append(
            rows, ld, int(col0), w, float(eps), None, None, None, None, 0, 0, 0,
            None, out, T, n, _DT[rows.dtype], _stream()), "rmsnorm_columns")
        self.launches += 1
        return out

    def concat_cast(self, a, b, dtype):
        """[a; b] along the columns, from two float32 tensors into `dtype`."""
        _need(a.dtype == torch.float32 and b.dtype == torch.float32 and a.shape == b.shape and a.is_contiguous()
              and b.is_contiguous(), "concat_cast: two float32 tensors of one shape")
        T, H = a.shape
        out = torch.empty(T, 2 * H, dtype=dtype, device=a.device)
        _check(self.lib.ifx_concat_cast(a, b, out, T, H, _DT[dtype], _stream()), "concat_cast")
        self.launches += 1
        return out

    def xielu(self, z, a_pos, a_neg):
        """a_pos z^2 + z/2 above zero, a_neg (e^z - 1 - z) + z/2 below, element by element, in float32."""
        splits, out_dtype = 1, z.dtype
        if isinstance(z, PartialSum):                      # a K-split product: the slices are added first, in the same pass
            out_dtype, splits, z = z.dtype, z.splits, z.parts
        _need(z.is_contiguous(), "xielu: contiguous input")
        out = torch.empty(tuple(z.shape[-2:]), dtype=out_dtype, device=z.device)
        _check(self.lib.ifx_xielu(z, out, (out.numel()), float(a_pos),
                                  float(a_neg), _DT[z.dtype], _DT[out_dtype], splits, _stream()), "xielu")
        self.launches += 1
        return out

    def softcap(self, logits, cap):
        """logits <- cap tanh(logits / cap), in place (float32)."""
        _need(logits.dtype == torch.float32 and logits.is_contiguous(), "softcap: float32 logits")
        _check(self.lib.ifx_softcap(logits, (logits.numel()), float(cap), _stream()),
               "softcap")
        self.launches += 1

    def short_conv(self, h, w, taps, state, index, ctx, add_input=True, bias=None, act=None, columns=None):
        """h + causal depthwise convolution of h over each request's tokens; `state[:, index]` (float32
        [slots, convolutions, taps - 1, channels]) brings the inputs before the step and takes the last ones.
        `add_input` False: the convolution alone; `bias` (float32 [channels]) is added and `act` ("silu") applied
        behind it; `columns` = (first, count): the convolution runs over those columns of `h` and returns them alone."""
        T, width = h.shape
        col0, C = (0, width) if columns is None else (int(columns[0]), int(columns[1]))
        _need(h.is_contiguous() and w.dtype == torch.float32 and tuple(w.shape) == (C, taps) and w.is_contiguous()
              and 0 <= col0 and col0 + C <= width and act in (None, "silu")
              and (bias is None or (bias.dtype == torch.float32 and bias.numel() == C)), "short_conv: bad operands")
        st_ptr, stride = 0, 0
        if taps > 1:
            _need(state is not None and state.dtype == torch.float32 and tuple(state.shape[2:]) == (taps - 1, C)
                  and state.stride(3) == 1 and state.stride(2) == C and 0 <= index < state.shape[1],
                  "short_conv: the state does not fit the convolution")
            stride = state.stride(0)                       # a slot's rows may be part of a longer state row
            st_ptr = state.data_ptr() + 4 * index * state.stride(1)
        out = torch.empty(T, C, dtype=h.dtype, device=h.device)
        _check(self.lib.ifx_short_conv_ex(h.data_ptr() + col0 * h.element_size(), width,
                                          w, bias, st_ptr, stride, ctx.token_req,
                                          ctx.req_slot, ctx.cu_seqlens, out, T, ctx.num_requests, C,
                                          taps, int(ctx.max_span > 1), float(1.0 if add_input else 0.0),
                                          int(act == "silu"), _DT[h.dtype], _stream()), "short_conv")
        self.launches += 1 + int(taps > 1 and ctx.max_span > 1)
        return out

    # -------------------------------------------------------- latent attention
    LATENT_PROMPT_MIN_ROWS = 64
    LATENT_TILE = 64           # tokens per work item of the tiled latent attention kernel

    def latent_attention_sections(self, ctx):
        """latent.items[P, 4] = (slot, first flat token, tokens, first position): every span in pieces of up
        to 64 tokens; a decoded token is an item of one."""
        items, base = [], 0
        for (start, n), slot in zip(ctx.spans, ctx.slots_host):
            for off in range(0, n, self.LATENT_TILE):
                items.extend((int(slot), base + off, min(self.LATENT_TILE, n - off), start + off))
            base += n
        return {"latent.items": items}

    def linear_heads(self, a, w, heads, k, n, w_is_nk, a_head_stride=None, out=None, out_head_stride=None):
        """One small product per head, heads side by side in the rows of `a` [T, >= heads * k]:
        out[:, h n:(h + 1) n] = a[:, h k:(h + 1) k] . W_h^T with W_h = w[h n:(h + 1) n] of [n, k] (w_is_nk), or
        a[:, h k:(h + 1) k] . W_h with W_h = w[h k:(h + 1) k] of [k, n].  bfloat16, through the library.
        `a_head_stride`: a head's columns begin that far apart in `a` (default k); `out` with `out_head_stride`:
        the heads' results go into columns of that tensor, that far apart."""
        T, lda = a.shape
        sa = k if a_head_stride is None else int(a_head_stride)
        _need(a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and a.is_contiguous() and w.is_contiguous(),
              "linear_heads: contiguous bfloat16 operands")
        _need(tuple(w.shape) == ((heads * n, k) if w_is_nk else (heads * k, n)) and sa >= k and lda >= (heads - 1) * sa + k,
              "linear_heads: shapes do not fit")
        so = n if out_head_stride is None else int(out_head_stride)
        if out is None:
            out = torch.empty(T, heads * so, dtype=torch.bfloat16, device=a.device)
        _need(out.dtype == torch.bfloat16 and out.is_contiguous() and out.shape[0] == T and so >= n
              and out.shape[1] >= (heads - 1) * so + n, "linear_heads: the output does not fit")
        ldw = k if w_is_nk else n
        _check(self.lib.ifx_gemm_cublas_bf16_batched(
            a, lda, sa, w, ldw, (k * n), out, out.shape[1], so, T, n, k, heads,
            int(bool(w_is_nk)), _stream()), "linear_heads")
        self.library_calls += 1
        return out

    def latent_norm_append(self, rows, col0, rank, w, eps, ctx, cache):
        """The latent of every token: columns col0 .. col0 + rank of `rows`, RMS-normed with weight `w`,
        written to the cache at the token's position."""
        T, ld = rows.shape
        kv, table = cache.kv, cache.block_table
        _need(kv is not None and table is not None and kv.dtype == rows.dtype, "latent_norm_append: no cache of the run's dtype")
        _need(kv.shape[1] == 1 and kv.shape[2] == 1 and kv.shape[4] == rank, "latent_norm_append: the cache is not one latent plane")
        write = bool(cache.writes)
        _check(self.lib.ifx_latent_norm_append(
            rows, ld, col0, w, float(eps), ctx.positions, ctx.token_req,
            ctx.req_slot, table, table.shape[1], cache.page_size, kv.shape[0], (kv if write else None),
            None, T, rank, _DT[rows.dtype], _stream()), "latent_norm_append")
        self.launches += 1

    def latent_rope_append(self, rows, col0, rank, rot, w, eps, q, heads, dim, rotary, ctx, cache, vdim=None, gate_col=None):
        """The cached row of every token: [columns col0 .. + rank of `rows`, RMS-normed with `w`; the `rot` columns
        behind them, turned by the token's position], written at the token's position.  Returns `q`
        [T, heads (dim + rot)] with every head's last `rot` elements turned the same way (in place), or, where the
        tiled attention kernel takes the sizes (`vdim` given), a `TurnedQueries`: the turned parts then lie in the
        rows of queries in latent space, [T, heads (rank + rot)], whose other columns `latent_attention` fills.  With
        `gate_col` returns (that, sigmoid of the `heads` columns of `rows` from gate_col on as float32 [T, heads])."""
        T, ld = rows.shape
        gate = None if gate_col is None else torch.empty(T, heads, dtype=torch.float32, device=rows.device)
        kv, table = cache.kv, cache.block_table
        _need(kv is not None and table is not None and kv.dtype == rows.dtype and q.dtype == rows.dtype,
              "latent_rope_append: no cache of the run's dtype")
        _need(kv.shape[1] == 1 and kv.shape[2] == 1 and kv.shape[4] == rank + rot,
              "latent_rope_append: the cache is not one plane of latent and turned part")
        _need(rows.is_contiguous() and q.is_contiguous() and q.shape[0] == T and q.shape[1] >= heads * (dim + rot),
              "latent_rope_append: contiguous rows")
        used, inter, mag, freq = 0, 0, 1.0, None
        if rot and rotary is not None:
            used, inter, mag, freq = int(rotary.rotary_dim), int(bool(rotary.interleaved)), float(rotary.magnitude), rotary.inv_freq
            _need(used <= rot and freq.dtype == torch.float32 and freq.numel() == used // 2,
                  "latent_rope_append: the table does not fit the turned part")
        write = bool(cache.writes)
        dst, ld_dst, head_stride, offset, result = q, q.shape[1], dim + rot, dim, q
        if (rot and vdim is not None and self.latent_tiles and rows.dtype == torch.bfloat16 and dim % 8 == 0 and vdim % 8 == 0
                and q.shape[1] % 8 == 0 and self.lib.ifx_latent_attention_mma_supports_rot(rank, rot)):
            dst = torch.empty(T, heads * (rank + rot), dtype=torch.bfloat16, device=rows.device)
            ld_dst, head_stride, offset, result = heads * (rank + rot), rank + rot, rank, TurnedQueries(q, dst)
        _check(self.lib.ifx_latent_rope_append(
            rows, ld, int(col0), w, float(eps), q, q.shape[1], dst, ld_dst, head_stride, offset,
            freq, used, inter, float(mag), ctx.positions, ctx.token_req, ctx.req_slot,
            table, table.shape[1], cache.page_size, kv.shape[0], (kv if write else None), T, rank, rot, heads, dim,
            gate, int(gate_col or 0), _DT[rows.dtype], _stream()), "latent_rope_append")
        self.launches += 1
        return result if gate_col is None else (result, gate)

    def latent_attention(self, q_rows, w_uk, w_uv, sinks, heads, dim, vdim, rank, window, scale, ctx, cache, rot=0,
                         head_gate=None):
        """Attention over cached latents (see csrc/latent_attention.cu).  `q_rows`: [T, >= heads * (dim + rot)], the
        queries in its first columns, every head's `rot` turned elements behind its `dim` plain ones; cached rows
        are [latent of `rank`; turned key part of `rot`].  `head_gate` (float32 [T, heads]) multiplies the heads' outputs.
        Returns [T, heads * vdim]."""
        turned = None
        if isinstance(q_rows, TurnedQueries):
            q_rows, turned = q_rows.rows, q_rows.latent
        T, ldq = q_rows.shape
        kv, table = cache.kv, cache.block_table
        _need(kv is not None and table is not None and kv.dtype == q_rows.dtype, "latent_attention: no cache of the run's dtype")
        _need(q_rows.is_contiguous() and w_uk.is_contiguous() and w_uv.is_contiguous(), "latent_attention: contiguous operands")
        _need(tuple(w_uk.shape) == (heads * dim, rank) and tuple(w_uv.shape) == (heads * vdim, rank),
              "latent_attention: the up-projections do not fit the sizes")
        _need(kv.shape[4] == rank + rot and ldq >= heads * (dim + rot), "latent_attention: rows do not hold the turned part")
        if turned is not None:
            return self._latent_attention_tiles(q_rows, w_uk, w_uv, sinks, heads, dim, vdim, rank, window, scale, ctx, cache,
                                                rot=rot, ql=turned, head_gate=head_gate)
        _need(head_gate is None or (head_gate.dtype == torch.float32 and tuple(head_gate.shape) == (T, heads)
                                    and head_gate.is_contiguous()), "latent_attention: a gate per head is float32 [tokens, heads]")
        tiled = (self.latent_tiles and not rot and q_rows.dtype == torch.bfloat16 and dim % 8 == 0 and vdim % 8 == 0
                 and ldq % 8 == 0 and self.lib.ifx_latent_attention_mma_supports(rank))
        if rot or (head_gate is not None and not tiled):
            out = torch.empty(T, heads * vdim, dtype=q_rows.dtype, device=q_rows.device)
            _check(self.lib.ifx_latent_attention_generic_rot(
                q_rows, ldq, w_uk, w_uv, sinks, kv, table, ctx.positions,
                ctx.token_req, ctx.req_slot, None, out, T, heads, dim, vdim, rank, cache.page_size,
                table.shape[1], kv.shape[0], 0 if window is None else int(window), float(scale), int(rot),
                head_gate, _DT[q_rows.dtype], _stream()), "latent_attention (turned part)")
            self.launches += 1
            return out
        if tiled:
            return self._latent_attention_tiles(q_rows, w_uk, w_uv, sinks, heads, dim, vdim, rank, window, scale, ctx, cache,
                                                head_gate=head_gate)
        out = torch.empty(T, heads * vdim, dtype=q_rows.dtype, device=q_rows.device)
        _check(self.lib.ifx_latent_attention_generic(
            q_rows, ldq, w_uk, w_uv, sinks, kv, table, ctx.positions,
            ctx.token_req, ctx.req_slot, None, out, T, heads, dim, vdim, rank, cache.page_size,
            table.shape[1], kv.shape[0], 0 if window is None else int(window), float(scale), _DT[q_rows.dtype],
            _stream()), "latent_attention")
        self.launches += 1
        return out

    def _latent_by_tma(self, rank, rot, page_size):
        """Whether the kernels whose tiles come by TMA take these sizes; asked of them once per sizes."""
        key = rank, rot, page_size
        if key not in self._latent_sizes:
            self._latent_sizes[key] = bool(self.lib.ifx_latent_decode_supports(*key) and self.lib.ifx_latent_prompt_supports(*key))
        return self._latent_sizes[key]

    def _latent_attention_tiles(self, q_rows, w_uk, w_uv, sinks, heads, dim, vdim, rank, window, scale, ctx, cache, rot=0,
                                ql=None, head_gate=None):
        """bfloat16: queries into latent space (a product per head), the tensor-core kernel over cached latents
        with all heads of a token tile in one block, the value projection per head on the weighted latents.
        With `rot`, `ql` [T, heads (rank + rot)] holds the turned query parts already, behind the columns that the
        product per head fills."""
        T = q_rows.shape[0]
        kv, table = cache.kv, cache.block_table
        if "latent.items" not in ctx.extra:                # a step context built without the mixer as a provider
            vals = self.latent_attention_sections(ctx)["latent.items"]
            ctx.extra["latent.items"] = torch.tensor(vals, dtype=torch.int32, device=q_rows.device)
            ctx.extra_len["latent.items"] = len(vals)
        items, num_items = ctx.extra["latent.items"], ctx.extra_len["latent.items"] // 4
        if rot:
            self.linear_heads(q_rows, w_uk, heads, dim, rank, w_is_nk=False, a_head_stride=dim + rot, out=ql,
                              out_head_stride=rank + rot)
        else:
            ql = self.linear_heads(q_rows, w_uk, heads, dim, rank, w_is_nk=False)           # [T, heads * rank]
        win = 0 if window is None else int(window)
        splits = 1
        max_keys = int(ctx.max_kv_len if not win else min(win, ctx.max_kv_len))
        by_tma = self._latent_by_tma(rank, int(rot), cache.page_size) and (ql.data_ptr() | kv.data_ptr()) % 16 == 0
        decode = by_tma and ctx.max_span == 1 and self.latent_decode
        if decode:                                         # decoded tokens only, a kernel of their own
            stretch = int(self.lib.ifx_latent_decode_stretch(T, heads, max_keys))
            splits = -(-(max_keys + 15) // stretch)        # (a window may begin inside a tile of 16 keys)
            decode = splits <= 64
        # spans of which a block's 128 rows (a token with all its heads) are a good part: the tcgen05 kernel
        # (whose running maximum is of the scores before they are scaled, so that a scale has to be positive)
        prompt = (by_tma and not decode and self.latent_prompt and scale > 0.0
                  and min(n for _s, n in ctx.spans) * heads >= self.LATENT_PROMPT_MIN_ROWS)
        if decode:
            pass
        elif prompt:                                       # a block an SM: cut the keys while there are fewer blocks than SMs
            # A part keeps two tiles of keys at least, and four from 25 blocks on, where adding the parts up takes as long as two
            # tiles (whole part, us, with two / four tiles: 300 tokens behind 500 of 12 heads, 29 blocks, 42.4 / 37.0, of 28 heads
            # 66.1 / 50.8; 500 tokens of 12, 47 blocks, 46.8 / 38.3; 100 behind 800, ten blocks, 42.0 / 45.4).
            blocks = sum(-(-n * heads // 128) for _s, n in ctx.spans)
            splits = max(1, min(148 // blocks, -(-max_keys // 128) // (2 if blocks <= 24 else 4), 16))
        elif ctx.max_span == 1:                            # cut the keys so that the SMs fill
            blocks = num_items * -(-heads // 64)                 # about four warps a SM, at least two key tiles each
            splits = max(1, min(592 // max(1, blocks), max_keys // 64, 64))
        else:
            # prompt portions: a block walks its keys tile after tile, and the last tokens' blocks walk all of them;
            # while the grid does not fill the SMs twice over (three blocks a SM), cut every block's keys in 2..4
            hc = min(heads, 64)
            qt = max(1, min(64 // hc, self.LATENT_TILE, ctx.max_span))
            blocks = -(-T // qt) * -(-heads // 64)
            splits = max(1, min(888 // max(1, blocks), max_keys // 256, 4))
        ws = None
        if splits > 1:
            ws = torch.empty(int(self.lib.ifx_latent_attention_mma_workspace(T * heads, rank, splits)), dtype=torch.uint8,
                             device=q_rows.device)
        olat = torch.empty(T, heads * rank, dtype=torch.bfloat16, device=q_rows.device)
        if decode:
            _check(self.lib.ifx_latent_decode(
                ql, kv, table, items, num_items, sinks, olat, ws, T, heads, rank, int(rot),
                cache.page_size, table.shape[1], kv.shape[0], win, float(scale), stretch, splits, head_gate,
                self.error_flag, _stream()), "latent_attention (decode)")
        elif prompt:
            _check(self.lib.ifx_latent_prompt(
                ql, kv, table, items, num_items, int(min(self.LATENT_TILE, ctx.max_span)), sinks,
                olat, ws, T, heads, rank, int(rot), cache.page_size, table.shape[1], kv.shape[0], win,
                float(scale), splits, head_gate, self.error_flag, _stream()), "latent_attention (prompt)")
        else:
            _check(self.lib.ifx_latent_attention_mma_rot(
                ql, kv, table, items, num_items, int(min(self.LATENT_TILE, ctx.max_span)), sinks,
                olat, ws, T, heads, rank, int(rot), cache.page_size, table.shape[1], kv.shape[0], win,
                float(scale), splits, head_gate, _stream()), "latent_attention (tiles)")
        self.launches += 1 + int(splits > 1)
        return self.linear_heads(olat, w_uv, heads, rank, vdim, w_is_nk=True)               # [T, heads * vdim]

    # ------------------------------------------------- recurrence with matrix state
    def cast_rows(self, x, dtype):
        """float32 rows in the run's dtype (the rows themselves when that is float32)."""
        if dtype == torch.float32:
            return x
        _need(x.dtype == torch.float32 and x.is_contiguous(), "cast_rows: contiguous float32 rows")
        out = torch.empty(x.shape, dtype=dtype, device=x.device)
        _check(self.lib.ifx_cast_rows(x, out, (x.numel()), _DT[dtype], _stream()), "cast_rows")
        self.launches += 1
        return out

    def tanh(self, z):
        """tanh of every element, in place."""
        _need(z.is_contiguous(), "tanh: contiguous input")
        _check(self.lib.ifx_tanh_rows(z, (z.numel()), _DT[z.dtype], _stream()), "tanh")
        self.launches += 1
        return z

    def token_shift_mix(self, x, mu, state, prev_offset, ctx, out_dtype):
        """mixes[m, t] = x[t] + (x[t - 1] - x[t]) * mu[m] for the float32 rows `x` [T, C] and `mu` [M, C]; the row
        before a span's first one is `state[slot, prev_offset : prev_offset + C]` (float32; zeros at a sequence's
        start).  The state is not changed here: `wkv_scan` leaves the step's last row there."""
        T, C = x.shape
        _need(x.dtype == torch.float32 and x.is_contiguous() and mu.dtype == torch.float32 and mu.is_contiguous()
              and mu.shape[1] == C, "token_shift_mix: float32 rows and weights of one width")
        _need(state is not None and state.dtype == torch.float32 and state.is_contiguous() and state.dim() == 2
              and prev_offset + C <= state.shape[1], "token_shift_mix: the state does not hold a row")
        out = torch.empty(mu.shape[0], T, C, dtype=out_dtype, device=x.device)
        _check(self.lib.ifx_token_shift_mix(
            x, mu, state.data_ptr() + 4 * prev_offset, state.shape[1],
            ctx.token_req, ctx.req_slot, ctx.cu_seqlens, out, T, C, mu.shape[0], _DT[out_dtype],
            _stream()), "token_shift_mix")
        self.launches += 1
        return out

    # Spans of this many tokens and more can go by stretches of 64 tokens in a bfloat16 run (csrc/chunk_scan.cu, delta_chunks.cu), of 128
    # with one decay per head (csrc/chunk_tcgen05.cu).  The other spans of the same step then go along, or through the scans token by
    # token in launches of their own: a stretch costs the same with one token as with all of them.
    CHUNK_SCAN_MIN_SPAN = 128

    def _long_spans(self, ctx):
        """(longest, tokens, number, stretches) of a step's spans of fewer than CHUNK_SCAN_MIN_SPAN tokens and the stretches of the others,
        found once a step; None for a context without a host list of spans, whose spans all go the same way."""
        got = getattr(ctx, "long_spans", None)
        if got is None and getattr(ctx, "spans", None):
            short = [n for _s, n in ctx.spans if n < self.CHUNK_SCAN_MIN_SPAN]
            got = ctx.long_spans = (max(short, default=0), sum(short), len(short), sum(-(-n // 64) for n in short),
                                    sum(-(-n // 64) for _s, n in ctx.spans if n >= self.CHUNK_SCAN_MIN_SPAN))
        return got

    stretch = 0                # tokens of a stretch of a decay per head: 64, 128, or 0 for the kernels' own rule

    def _stretch_beside(self, ctx, heads, dv):
        """The same where short spans go through the scan: the kernels' rule (ifx_chunk_scan_takes_128), which knows a step's tokens alone, of
        the long spans' stretches.  us, 24 heads of 128 x 64, 300 tokens beside eight spans of 100: 171 by 64, 180 by 128."""
        return 128 if self._long_spans(ctx)[4] * heads * (dv // 64) > 148 else 64

    def _scans_by_chunks(self, dtype, ctx, heads, dk, dv, *rows, constant=False):
        """Which of a recurrence's spans go by stretches of tokens: False, none; else (the fewest tokens of one that does, the most
        tokens of one that does not or 0).  Where that pays, with sizes the kernels are made for, rows on 16-byte boundaries (those
        given here; the kernels look at theirs themselves), and in a bfloat16 run (the order of the sums then depends on how a span
        was cut into steps)."""
        if not (self.chunk_scans and dtype is torch.bfloat16 and ctx.max_span >= self.CHUNK_SCAN_MIN_SPAN):
            return False
        if dk not in (64, 128) or dv % 64 or ctx.num_requests > 64:              # ifx_chunk_scan_supports, without a call
            return False
        spans = self._long_spans(ctx)
        plan = (1, 0) if spans is None else self.stretches_pay(ctx.max_span, heads * dv // 64, constant and dk == 64, *spans)
        return plan if plan and all(t.data_ptr() % 16 == 0 and (t.dim() < 2 or t.stride(0) % 4 == 0) for t in rows) else False

    @classmethod
    def stretches_pay(cls, longest, blocks, cheap, short, short_tokens, short_spans, short_stretches, stretches):
        """The plan for a step whose longest span has `longest` tokens, with `blocks` blocks a stretch.  Short spans go along where their
        stretches (0.13 us a block of 64 tokens) take less than a launch of the scan for them.  Otherwise what is gained is the time between
        the longest span and the longest short one.  us, the scan alone and all by stretches (the long ones beside the scan), 12 heads of
        128 x 128 with a constant decay; wkv, 24 heads of 64: 128 tokens 40 / 30; 39 / 28; sixteen of 128 212 / 92; 183 / 143; 128 and 20
        46 / 31 (41); 43 / 29 (39); 228 and 100 79 / 36 (73); 71 / 39 (72); 128 and 31 of one token 75 / 149 (63); 95 / 135 (60); 512 and
        31 of one token 223 / 152 (69); 260 / 151 (74); 512, 100, 80 and 29 of one token 234 / 154 (107); 267 / 154 (122).  At 56 and 28
        heads 128 and 31 of one token 154 / 285 (105) and 124 / 367 (109), but 63 of one token 28 heads of 128 x 128 188 / 896 (194): what the
        launch for very many states costs has to be gained.  `cheap`, a constant decay and keys of 64 numbers, whose scan wins over
        stretches of 64 where very many are of short spans.  The lines were drawn for stretches of 64 tokens, which wkv and decays per
        channel have; no step of 330 measured ones takes 5 % longer than the scan alone.  Stretches of 128 take about half as long, so that more steps with a
        decay per head would gain: 300 and eight of 100 tokens 174 / 55 (138); `cheap`, 28 heads, 32 of 128 441 / 300."""
        if cheap and stretches > 24 + longest // 4:
            return False
        if 0.13 * short_stretches * blocks <= 8 + 0.22 * short + 0.035 * short_spans * blocks:
            return 1, 0
        beside = longest >= short + 128 or (short < 24 and (longest >= 192 or short_spans * blocks <= 2500))
        return (cls.CHUNK_SCAN_MIN_SPAN, short) if beside else False

    def wkv_scan(self, r, k, v, w_raw, g, w0, u, norm_w, eps, heads, dim, state, prev_offset, x, ctx, out_dtype):
        """The recurrence of csrc/wkv.cu over every request's tokens.  r, k, v, w_raw, g: float32 [T, heads * dim], each
        contiguous or a column block of a wider matrix (all with the same distance between rows);
        `state`: float32 [slots, heads * dim * dim + C], the matrices first, then the last input row, both moved on.
        Returns out / rms(out) per head * norm_w * silu(g) in `out_dtype`."""
        T, HD = r.shape
        C = x.shape[1]
        ld, ld_w = max(int(r.stride(0)), HD), max(int(w_raw.stride(0)), HD)
        for t in (r, k, v, w_raw, g):
            _need(t.dtype == torch.float32 and tuple(t.shape) == (T, HD) and t.stride(1) == 1
                  and (T == 1 or t.stride(0) == (ld_w if t is w_raw else ld)),
                  "wkv_scan: float32 [T, heads * dim] inputs; r, k, v and g with one distance between rows")
        for t in (w0, u, norm_w):
            _need(t.dtype == torch.float32 and t.is_contiguous() and t.numel() == HD, "wkv_scan: float32 constants of heads * dim")
        _need(HD == heads * dim and prev_offset == heads * dim * dim and state.dtype == torch.float32 and state.is_contiguous()
              and state.dim() == 2 and state.shape[1] == prev_offset + C and x.dtype == torch.float32 and x.is_contiguous(),
              "wkv_scan: the state does not fit the sizes")
        by_chunks, size = self._scans_by_chunks(out_dtype, ctx, heads, dim, dim), T * HD
        if by_chunks:
            least, short = by_chunks
            size += int(self.lib.ifx_chunk_scan_scratch_floats(T, ctx.num_requests, least, heads, dim, dim, 1))
        scratch = torch.empty(size, dtype=torch.float32, device=r.device)         # the sums, and what the stretches need
        y = torch.empty(T, HD, dtype=out_dtype, device=r.device)
        common = (state, state.data_ptr() + 4 * prev_offset, state.shape[1], x, C, ctx.cu_seqlens,
                  ctx.req_slot, scratch)
        rows = (r, k, v, w_raw)
        if by_chunks:
            room = scratch.data_ptr() + 4 * T * HD               # (heads of 64 or 128: still on 16 bytes)
            rc = self.lib.ifx_chunk_wkv_scan(*rows, w0, u, *common, ctx.num_requests, T, least, heads, dim, ld, ld_w, room,
                                             _stream())
            if rc != _MISALIGNED:
                _check(rc, "wkv_scan (stretches)")
                if short:
                    _check(self.lib.ifx_wkv_scan(*rows, g, w0, u, norm_w, float(eps), *common, y,
                                                 ctx.num_requests, T, heads, dim, ld, ld_w, _DT[out_dtype], short, _stream()),
                           "wkv_scan (short spans)")
                    self.launches += 1
                _check(self.lib.ifx_wkv_norm(scratch, g, norm_w, float(eps), y, T, heads, dim, ld,
                                             _DT[out_dtype], _stream()), "wkv_norm")
                self.launches += 4
                return y
        _check(self.lib.ifx_wkv_scan(*rows, g, w0, u, norm_w, float(eps), *common, y, ctx.num_requests,
                                     T, heads, dim, ld, ld_w, _DT[out_dtype], 0, _stream()), "wkv_scan")
        self.launches += 1
        return y

    def _delta_by_chunks(self, dtype, ctx, tokens, heads, dim):
        """Which spans of the delta rule go by stretches, as above."""
        if not (self.chunk_scans and dtype is torch.bfloat16 and ctx.max_span >= self.CHUNK_SCAN_MIN_SPAN):
            return False
        if dim != 64 or ctx.num_requests > 64:                                   # ifx_delta_chunks_supports, without a call
            return False
        spans = self._long_spans(ctx)
        if spans is None:
            return tokens <= 8 * ctx.max_span and (1, 0)
        return self.delta_stretches_pay(heads, tokens, ctx.num_requests, ctx.max_span, *spans)

    @classmethod
    def delta_stretches_pay(cls, heads, tokens, requests, longest, short, short_tokens, short_spans, short_stretches, stretches):
        """A stretch of the delta rule does several times a token's work of the scan; what is gained is that the tokens of one span run
        side by side, so this compares what the ways take: the scan for all, stretches for all, stretches for the long spans beside
        the scan for the others.  us, fitted to what follows within a sixth: the scan walks its longest span at 0.3 a token and more
        with more columns at once; the stretches go in rounds of 148 blocks (a head's stretch each), every block walks the requests, each
        span behind the eighth costs its heads' carries, and beyond 3,000 blocks what they hand on (40 KB each) does not stay in L2.
        us, 24 heads of 64, the scan alone and the stretches for all (for the long ones beside the scan): 128 tokens 46 / 32; 256 85 / 34;
        512 164 / 60; 2,048 658 / 193; two of 256 98 / 61; four of 256 125 / 93; four of 512 261 / 190; eight of 512 368 / 341; eight of 128
        92 / 101; sixteen of 150 224 / 260; 128 and 31 of one token 66 / 181 (58, left: what it gains is within the fit's error); 512 and 31
        of one token 216 / 221 (89), 63 228 / 469 (111); 256 and 100 94 / 40 (80); four spans of 512, 100, 80 and 29 212 / 87 (114).
        56 heads: 128 56 / 38; 256 104 / 62; 2,048 833 / 396; four of 256 265 / 219; four of 512 516 / 394; sixteen of 128 420 / 469,
        thirty-two 794 / 1,013; sixteen of 256 817 / 833; 512 and 31 of one token 297 / 560 (183), 63 321 / 1,196 (230, left)."""
        def scan(longest, tokens, requests):
            columns = tokens * heads / longest             # heads at work at once, on average
            return longest * max(0.3 + 0.0019 * columns, columns / 275) + 0.018 * requests * heads

        def chunks(blocks, spans):
            return (20.6 * -(-blocks // 148) + 0.6 * (longest / 64) + 0.07 * blocks + 4 + 1.5 * max(0, requests - 4)
                    + 0.06 * heads * max(0, spans - 8) + 0.1 * max(0, blocks - 3000))
        least, alone = 1, 6 + scan(longest, tokens, requests - 1)
        best = chunks((stretches + short_stretches) * heads, requests)
        if short:
            beside = chunks(stretches * heads, requests - short_spans) + 10 + scan(short, short_tokens, short_spans)
            if beside < best:
                least, best = cls.CHUNK_SCAN_MIN_SPAN, beside
        return best < alone and (least, short if least > 1 else 0)

    def delta_rule_scan(self, proj, w_raw, w0, a_bias, norm_w, eps, heads, dim, state, ctx, out_dtype):
        """The recurrence of csrc/delta_rule.cu over every request's tokens.  `proj`: float32 [T, 5 heads dim], the
        projections r, k, v, g, a side by side; `w_raw`: float32 [T, heads dim]; `state`: float32 [slots, >= heads dim
        dim] (rows may be further apart), the matrices [head, key channel, value channel], moved on.  Returns
        out / rms(out) per head * norm_w * sigmoid(g) in `out_dtype`."""
        T, HD = proj.shape[0], heads * dim
        _need(proj.dtype == torch.float32 and proj.is_contiguous() and proj.shape[1] >= 5 * HD and w_raw.dtype == torch.float32
              and w_raw.is_contiguous() and tuple(w_raw.shape) == (T, HD), "delta_rule_scan: float32 projections")
        for t in (w0, a_bias, norm_w):
            _need(t.dtype == torch.float32 and t.is_contiguous() and t.numel() == HD, "delta_rule_scan: float32 constants of heads * dim")
        _need(state is not None and state.dtype == torch.float32 and state.dim() == 2 and state.stride(1) == 1
              and state.shape[1] >= HD * dim, "delta_rule_scan: the state does not fit the sizes")
        y = torch.empty(T, HD, dtype=out_dtype, device=proj.device)
        by_chunks = self._delta_by_chunks(out_dtype, ctx, T, heads, dim)
        if by_chunks:
            least, short = by_chunks
            room = torch.empty(int(self.lib.ifx_delta_chunks_scratch_floats(T, ctx.num_requests, least, heads)), dtype=torch.float32,
                               device=proj.device)
            scan_room = None
            if short:
                scan_room = torch.empty(int(self.lib.ifx_delta_rule_scratch_floats(T, heads, dim)), dtype=torch.float32, device=proj.device)
            rc = self.lib.ifx_delta_chunks_scan(
                proj, proj.shape[1], w_raw, w0, a_bias, norm_w, float(eps), state,
                state.stride(0), ctx.cu_seqlens, ctx.req_slot, room, y, ctx.num_requests, T,
                least, heads, dim, _DT[out_dtype], scan_room, self.error_flag, _stream())
            if rc != _MISALIGNED:
                _check(rc, "delta_rule_scan (stretches)")
                self.launches += 6 if short else 4
                return y
        scratch = torch.empty(int(self.lib.ifx_delta_rule_scratch_floats(T, heads, dim)), dtype=torch.float32, device=proj.device)
        _check(self.lib.ifx_delta_rule_scan(
            proj, proj.shape[1], w_raw, w0, a_bias, norm_w, float(eps), state,
            state.stride(0), ctx.cu_seqlens, ctx.req_slot, scratch, y,
            ctx.num_requests, T, heads, dim, _DT[out_dtype], _stream()), "delta_rule_scan")
        self.launches += 3
        return y

    # ------------------------------------------------------- mixture of experts
    def moe_route(self, z, correction, top, of_chosen=False, kind=None, floor=0.0):
        """(ids int32 [T, top], weights float32 [T, top]) from router logits z float32 [T, n]: softmax scores; the
        `top` largest of score + correction are chosen, their weights are the scores.  `of_chosen`: the `top`
        largest of z + correction are chosen, and the weights are the softmax over the chosen logits alone.
        `kind` = "sigmoid_normalized": scores = sigmoid(z), the `top` largest of score + correction are chosen, and the
        weights are the chosen scores divided by (their sum + floor)."""
        _need(kind in (None, "sigmoid_normalized"), f"moe_route: unknown kind {kind!r}")
        T, n = z.shape
        _need(z.dtype == torch.float32 and z.is_contiguous() and (correction is None or (correction.dtype == torch.float32
              and correction.numel() == n)), "moe_route: float32 logits and corrections")
        ids = torch.empty(T, top, dtype=torch.int32, device=z.device)
        weights = torch.empty(T, top, dtype=torch.float32, device=z.device)
        _check(self.lib.ifx_moe_route_kind(z, correction, ids, weights, T, n, int(top),
                                           2 if kind == "sigmoid_normalized" else int(bool(of_chosen)), float(floor),
                                           _stream()), "moe_route")
        self.launches += 1
        return ids, weights

    @staticmethod
    def _one_launch_router(T, K, n):
        """Whether router and choice in one launch take less than the library's product and the choice behind it.  The kernel has 16 tokens
        a block, so up to 2,368 tokens run at once, and each block reads the whole router; the library is slow for outputs that are no
        multiple of eight.  Up to 2,368 tokens the router's sizes alone decide, so that a token's choice depends on nothing else in the step.
        us, the two ways: 16 outputs, 24 tokens of 1,536 7.2 / 3.4, 4,096 of 2,880 11.8 / 9.1, 8,192 of 7,168 30.7 / 48.7; 24, 2,368 of 3,584
        10.4 / 9.0, 2,369 10.4 / 13.8, 24 of 7,168 13.3 / 11.3 (but 2 to 16 of them 8.8 / 10.4: the library has a kernel for those); 20, 4,096
        of 3,584 22.2 / 15.5; 64, 64 of 768 6.6 / 5.5, of 1,536 7.6 / 7.5, of 2,048 8.1 / 9.3, of 7,168 14.0 / 22.9; 33, 64 of 2,048 10.0 / 8.8,
        of 7,168 13.0 / 19.9.  (Router in L2.  Behind experts that push it out, layers of 18 outputs of 3,584 and up to 16 tokens take 1 % longer in one
        launch, 149.4 / 150.8, all others less or the same: 24 tokens 189.9 / 187.5, 16 outputs of 1,536 and 8 tokens 77.0 / 73.5.)"""
        odd = n % 8 != 0
        if T <= 2368:
            return n <= 32 or (n <= 64 and K <= (2048 if odd else 1536))
        return T <= 4736 and (n <= 8 or (n <= 16 and (odd or K <= 3072)) or (n <= 32 and (odd or K <= 512)))

    def moe_choose(self, h, w_router, correction, top, of_chosen=False, kind=None, floor=0.0):
        """`moe_route` of the router's logits h . w_router^T.  A bfloat16 router of up to 64 outputs takes one launch for both where that
        takes less."""
        n = w_router.shape[0]
        if not (h.dtype == w_router.dtype == torch.bfloat16 and self._one_launch_router(*h.shape, n) and h.is_contiguous() and w_router.is_contiguous()
                and h.shape[1] == w_router.shape[1] and h.shape[1] % 8 == 0 and (h.data_ptr() | w_router.data_ptr()) % 16 == 0):
            return self.moe_route(self.linear(h, w_router, out_dtype=torch.float32), correction, top, of_chosen=of_chosen, kind=kind, floor=floor)
        _need(kind in (None, "sigmoid_normalized"), f"moe_choose: unknown kind {kind!r}")
        _need(correction is None or (correction.dtype == torch.float32 and correction.is_contiguous() and correction.numel() == n),
              "moe_choose: float32 corrections")
        T = h.shape[0]
        ids = torch.empty(T, top, dtype=torch.int32, device=h.device)
        weights = torch.empty(T, top, dtype=torch.float32, device=h.device)
        _check(self.lib.ifx_moe_choose(h, w_router, correction, ids, weights, T, h.shape[1], n, int(top),
                                       2 if kind == "sigmoid_normalized" else int(bool(of_chosen)), float(floor), _stream()),
               "moe_choose")
        self.launches += 1
        return ids, weights

    def moe_experts(self, h, w_up, w_down, ids, weights, experts, out_dtype, glu=None):
        """sum over a token's choices of weight * W_down[e] relu(W_up[e] h)^2, or weight * h for e >= experts.
        w_up [experts, ff, width], w_down [experts, width, ff] in h's dtype.  `glu` = (limit, slope): w_up is
        [experts, 2 ff, width], an expert's gate rows above its up rows, and the activation is
        g sigmoid(slope g) (u + 1) with g = min(gate, limit), u = clamp(up, -limit, limit); a third number replaces
        the 1 (limit inf, slope 1 and 0 give silu(gate) * up)."""
        T, width = h.shape
        top = ids.shape[1]
        if glu is not None and len(glu) == 2:
            glu = (glu[0], glu[1], 1.0)
        if glu is not None:
            _need(experts > 0 and w_up.shape[1] % 2 == 0, "moe_experts: gated experts need gate and up rows")
            ff = w_up.shape[1] // 2
            _need(h.is_contiguous() and w_up.dtype == h.dtype and w_down.dtype == h.dtype and w_up.is_contiguous()
                  and w_down.is_contiguous() and tuple(w_up.shape) == (experts, 2 * ff, width)
                  and tuple(w_down.shape) == (experts, width, ff), "moe_experts: stacked expert weights in the activations' dtype")
            if h.dtype == torch.bfloat16:
                way = self.moe_kernels(T * top, int(experts), width, ff, True)
                if way != "tokens" and self._moe_on_tensor_cores(h, w_up, w_down, ff, width):
                    return (self._moe_experts_tiles if way == "tiles" else self._moe_experts_stream)(
                        h, w_up, w_down, ids, weights, experts, out_dtype, glu=glu)
            act = torch.empty(T * top, ff, dtype=h.dtype, device=h.device)
            out = torch.empty(T, width, dtype=out_dtype, device=h.device)
            _check(self.lib.ifx_moe_experts_glu(h, w_up, w_down, ids, weights, act, out,
                                                T, top, int(experts), width, ff, _DT[h.dtype], _DT[out_dtype], 1,
                                                float(glu[0]), float(glu[1]), float(glu[2]),
                                                _stream()), "moe_experts (gated)")
            self.launches += 2
            return out
        ff = w_up.shape[1] if experts else 1
        _need(h.is_contiguous() and (not experts or (w_up.dtype == h.dtype and w_down.dtype == h.dtype and w_up.is_contiguous()
              and w_down.is_contiguous() and tuple(w_up.shape) == (experts, ff, width) and tuple(w_down.shape) == (experts, width, ff))),
              "moe_experts: stacked expert weights in the activations' dtype")
        if experts and h.dtype == torch.bfloat16:
            way = self.moe_kernels(T * top, int(experts), width, ff, False)
            if way != "tokens" and self._moe_on_tensor_cores(h, w_up, w_down, ff, width):
                return (self._moe_experts_tiles if way == "tiles" else self._moe_experts_stream)(
                    h, w_up, w_down, ids, weights, experts, out_dtype)
        act = torch.empty(T * top, ff, dtype=h.dtype, device=h.device)
        out = torch.empty(T, width, dtype=out_dtype, device=h.device)
        _check(self.lib.ifx_moe_experts(h, (w_up if experts else None), (w_down if experts else None), ids,
                                        weights, act, out, T, top, int(experts), width, ff, _DT[h.dtype],
                                        _DT[out_dtype], _stream()), "moe_experts")
        self.launches += 2 if experts else 1
        return out

    # Which kernels make the experts of a bfloat16 step, by the number of (token, choice) pairs: per token, or, once the work is
    # MOE_TOKENS_MAX_WORK multiply-adds or there are MOE_TOKENS_MAX_PAIRS pairs, over rows sorted by expert, where every chosen
    # expert's weights are read once.  Measured on a B200, weights of two layers in turn (us, per token / sorted rows):
    #     4 experts, 2,048 x 2,048, one a token           1 token (8M) 21 / 31, 4 (34M): 21 / 31, 16 (134M): 52 / 30, 64: 137 / 30
    #     8 experts, 1,536 x 2,240 gated, two a token     1 token (21M) 38 / 25, 2 (41M): 42 / 31, 8: 63 / 43, 32: 166 / 44
    #    16 experts, the same, one a token                1 token (10M) 19 / 22, 2 (21M): 19 / 22, 4 (41M): 30 / 27, 8: 45 / 40
    #    16 experts, the same, four a token               1 token (41M) 61 / 31, 4: 85 / 53, 24: 243 / 70
    #    64 experts, 1,536 x 512, four a token            1 token (6M) 17 / 21, 4 (25M): 25 / 25, 8 (50M): 31 / 31, 16: 48 / 42
    #    64 experts, 2,048 x 1,408 gated, six a token     1 token (52M) 70 / 40, 4: 111 / 88
    #   256 experts, 2,048 x 1,024 gated, eight a token   1 token (50M) 64 / 42, 4: 103 / 94, 16: 282 / 221
    #    16 experts, 3,584 x 4,736 gated, four a token    1 token (204M) 153 / 88, 8: 520 / 257
    # Of the sorted rows, steps of few pairs an expert ("stream") cut the second product's K into slices and take the exact
    # exponential and division; the others ("tiles") do not.  A result's bits depend on that line, which lies where a kernel of its
    # own for few pairs was slower than tiles; the time does so little (the last row 252 instead of 257).
    MOE_TILES_MIN_PAIRS = 192
    MOE_TILES_LARGE_EXPERT = 1 << 23
    MOE_TOKENS_MAX_WORK = 40_000_000
    MOE_TOKENS_MAX_PAIRS = 512
    MOE_MAX_EXPERTS = 1024     # of sorted rows

    @classmethod
    def moe_kernels(cls, pairs, experts, width, ff, gated):
        """"tokens", or over sorted rows "stream" or "tiles"."""
        if pairs >= cls.MOE_TOKENS_MAX_PAIRS:
            return "tiles"
        if experts > cls.MOE_MAX_EXPERTS or pairs * ff * width * (3 if gated else 2) < cls.MOE_TOKENS_MAX_WORK:
            return "tokens"
        if ((pairs >= cls.MOE_TILES_MIN_PAIRS and pairs >= 12 * experts)
                or (ff * width >= cls.MOE_TILES_LARGE_EXPERT and pairs >= 2 * experts)):
            return "tiles"
        return "stream"

    @staticmethod
    def _moe_on_tensor_cores(h, w_up, w_down, ff, width):
        return (h.shape[0] > 0 and h.dtype == torch.bfloat16 and width % 8 == 0 and ff % 8 == 0 and h.data_ptr() % 16 == 0
                and w_up.data_ptr() % 16 == 0 and w_down.data_ptr() % 16 == 0
                and os.environ.get("INFERFLUX_B200_MOE_TILES", "1") != "0")

    def _moe_experts_stream(self, h, w_up, w_down, ids, weights, experts, out_dtype, glu=None):
        """bfloat16, few tokens: over sorted rows too, but K of the second product in up to three slices whose sums are added in
        float32, and a gate's exponential and division are not the fast ones."""
        return self._moe_experts_tiles(h, w_up, w_down, ids, weights, experts, out_dtype, glu=glu, few=True)

    def _moe_experts_tiles(self, h, w_up, w_down, ids, weights, experts, out_dtype, glu=None, few=False):
        """bfloat16: pairs sorted by expert, two tcgen05 products over the sorted rows by pairs of SMs (the
        activation, relu^2 or the gated one of `glu`, in the first one's epilogue), then the weighted sum per token."""
        T, width = h.shape
        top, ff = ids.shape[1], w_up.shape[1] // (2 if glu is not None else 1)
        room = self.lib.ifx_moe_sorted_scratch(T, top, int(experts), width, ff, int(few))
        scratch = torch.empty(room, dtype=torch.uint8, device=h.device)
        out = torch.empty(T, width, dtype=out_dtype, device=h.device)
        limit, slope, offset = (glu if len(glu) > 2 else (*glu, 1.0)) if glu is not None else (0.0, 0.0, 0.0)
        _check(self.lib.ifx_moe_sorted(h, w_up, w_down, ids, weights, out, T, top, int(experts),
                                       width, ff, _DT[out_dtype], int(glu is not None), int(few), float(limit),
                                       float(slope), float(offset), scratch, room, self.error_flag,
                                       _stream()), "moe experts (sorted rows)")
        self.launches += 5
        return out

    # ------------------------------------------- pairs of mixers, scans with a decayed matrix state
    def bigram_add(self, x, table, token_ids, state, mul_prev, mul_cur, buckets, vocab, ctx):
        """x[t] += table[(token before * mul_prev + token * mul_cur) mod buckets], the last row (`buckets`) at position 0;
        the token before a span's first one is state[slot, 0] (int32), which then takes the span's last token."""
        T, H = x.shape
        _need(x.dtype == torch.float32 and x.is_contiguous() and table.is_contiguous() and tuple(table.shape) == (buckets + 1, H)
              and state is not None and state.dtype == torch.int32, "bigram_add: bad operands")
        _check(self.lib.ifx_bigram_add(x, table, token_ids, ctx.positions, ctx.token_req,
                                       ctx.req_slot, ctx.cu_seqlens, state, state.stride(0),
                                       T, H, int(vocab), mul_prev, mul_cur, int(buckets),
                                       _DT[table.dtype], _stream()), "bigram_add")
        self.launches += 1

    def rmsnorm_pair(self, x, w_a, eps_a, w_b, eps_b, out_dtype, delta=None, vectors=None):
        """x += delta (if any); two RMS norms of the same float32 rows, one kernel.  `vectors` (a.s_a, b, s_b, b2 as in
        residual_add_vectors): x += s_a * a + s_b * (b + b2) in the same kernel."""
        if delta is not None:
            self.residual_add(x, delta)
        T, H = x.shape
        va = vb = vb2 = vsa = vsb = None
        if vectors is not None:
            va, vsa, vsb = self.materialize(vectors.a), vectors.s_a, vectors.s_b
            vb = None if vectors.b is None else self.materialize(vectors.b)
            vb2 = None if vectors.b2 is None else self.materialize(vectors.b2)
            if vb is not None and vb2 is not None and vb2.dtype != vb.dtype:
                vb2 = vb2.to(vb.dtype)
            _need(va.shape == x.shape and va.is_contiguous() and (vb is None or (vb.shape == x.shape and vb.is_contiguous()))
                  and (vb2 is None or (vb is not None and vb2.is_contiguous())), "rmsnorm_pair: the sum's rows do not fit")
        _need(x.dtype == torch.float32 and x.is_contiguous() and w_a.numel() == H and w_b.numel() == H
              and w_a.dtype == torch.float32 and w_b.dtype == torch.float32, "rmsnorm_pair: bad operands")
        out_a = torch.empty(T, H, dtype=out_dtype, device=x.device)
        out_b = torch.empty(T, H, dtype=out_dtype, device=x.device)
        _check(self.lib.ifx_rmsnorm_pair(x, w_a, float(eps_a), w_b, float(eps_b), out_a,
                                         out_b, T, H, _DT[out_dtype], va, _DT[va.dtype] if va is not None else 0,
                                         vsa, vb, vb2, _DT[vb.dtype] if vb is not None else 0, vsb,
                                         _stream()), "rmsnorm_pair")
        self.launches += 1
        return out_a, out_b

    def gate_mul(self, a, g, kind):
        """a * sigmoid(g) (`sigmoid`) or a * silu(g) (`silu`), in a's dtype."""
        _need(kind in ("sigmoid", "silu") and a.shape == g.shape and a.dtype == g.dtype and a.is_contiguous() and g.is_contiguous(),
              "gate_mul: bad operands")
        out = torch.empty_like(a)
        _check(self.lib.ifx_gate_mul(a, g, out, (a.numel()), _DT[a.dtype], int(kind == "silu"),
                                     _stream()), "gate_mul")
        self.launches += 1
        return out

    @staticmethod
    def _rows_f32(t, what):
        if t.dtype != torch.float32 or t.dim() != 2 or t.stride(1) != 1:
            raise KernelError(f"{what}: float32 rows with unit column stride")
        return t.data_ptr(), t.stride(0)

    def decay_scan(self, q, k, v, raw, state, ctx, heads, groups, dk, dv, decay, tau=1.0, q_scale=1.0, step_bias=None,
                   log_rate=None, skip=None, rate=None):
        """Per request and head a float32 matrix S, kept in `state` [slots, >= heads dv dk] as [head, value channel, key
        channel]: S <- diag(w_t) S + k_t v_t^T, o_t = S^T (q_scale q_t) with the new S.  q, k: float32 [T, groups dk]
        (head h reads group h // (heads / groups)); v: [T, heads dv]; rows may be slices of wider rows.  Returns
        float32 [T, heads dv].
        decay `sigmoid_root`: raw [T, heads dk], w = sigmoid(raw)^(1/tau).
        decay `softplus_step`: raw [T, heads], dt = softplus(raw + step_bias), w = exp(-exp(log_rate) dt) for the whole
        head, k is multiplied by dt, and skip[h] v_t is added to o_t.
        decay `constant`: raw None, w = rate[h] whatever the token."""
        T = q.shape[0]
        mode = _DECAYS.get(decay)
        if mode is None:
            raise KernelError(f"decay_scan: unknown decay {decay!r}")
        _need((raw is None) == (mode == 2) == (rate is not None), "decay_scan: a constant decay comes from `rate`, any other from `raw`")
        _need(q.shape[1] == groups * dk and k.shape[1] == groups * dk and v.shape[1] == heads * dv
              and k.shape[0] == T and v.shape[0] == T
              and (raw is None or tuple(raw.shape) == (T, heads * dk if mode == 0 else heads)),
              "decay_scan: the rows do not fit the head counts")
        _need(state is not None and state.dtype == torch.float32 and state.stride(1) == 1 and state.shape[1] >= heads * dv * dk,
              "decay_scan: the state does not fit the heads")
        for vec in (step_bias, log_rate, skip, rate):
            _need(vec is None or (vec.dtype == torch.float32 and vec.numel() == heads and vec.is_contiguous()),
                  "decay_scan: per-head vectors are float32 [heads]")
        out = torch.empty(T, heads * dv, dtype=torch.float32, device=q.device)
        rows = (*self._rows_f32(q, "decay_scan q"), *self._rows_f32(k, "decay_scan k"), *self._rows_f32(v, "decay_scan v"),
                *(self._rows_f32(raw, "decay_scan raw") if raw is not None else (None, 0)), state, state.stride(0),
                ctx.req_slot, ctx.cu_seqlens, out, step_bias, log_rate, skip)
        longest = int(ctx.max_span)
        by_chunks = self._scans_by_chunks(getattr(ctx, "dtype", None), ctx, heads, dk, dv, constant=mode == 2)
        if by_chunks:
            least, short = by_chunks
            room = torch.empty(int(self.lib.ifx_chunk_scan_scratch_floats(T, ctx.num_requests, least, heads, dk, dv, int(mode == 0))),
                               dtype=torch.float32, device=q.device)
            stretch = self.stretch or (self._stretch_beside(ctx, heads, dv) if short else 0)
            rc = self.lib.ifx_chunk_decay_scan(*rows, ctx.num_requests, T, least, int(heads), int(groups), int(dk), int(dv), mode,
                                               float(tau), float(q_scale), room, rate,
                                               stretch, self.error_flag, _stream())
            if rc != _MISALIGNED:
                _check(rc, "decay_scan (stretches)")
                self.launches += 3
                if not short:
                    return out
                longest = short                            # the other spans, token by token
        scratch = None                                     # steps with long spans make their decays in a pass of their own
        if longest >= 64 and mode != 2:
            scratch = torch.empty(T * (heads * dk if mode == 0 else 2 * heads), dtype=torch.float32, device=q.device)
        _check(self.lib.ifx_decay_scan_rate(*rows, ctx.num_requests, T, longest, int(longest < ctx.max_span), int(heads), int(groups), int(dk),
                                            int(dv), mode, float(tau), float(q_scale), 296, scratch, rate, _stream()),
               "decay_scan")
        self.launches += 1 + int(scratch is not None)
        return out

    def gated_groupnorm(self, y, gate, w, eps, groups, gate_first, out_dtype, kind="silu"):
        """Rows of y (float32 [T, C]) in `groups` equal parts, each over its own root mean square, times w (of size C, or
        of a part's size and then the same for every part; None: no weight) and silu(gate) (float32 rows, maybe a slice of wider ones):
        the gate multiplies before the norm (`gate_first`) or behind it.  `kind` "sigmoid": sigmoid(gate) in its place."""
        T, C = y.shape
        _need(y.dtype == torch.float32 and y.is_contiguous() and tuple(gate.shape) == (T, C) and C % groups == 0
              and (w is None or (w.dtype == torch.float32 and w.is_contiguous() and w.numel() in (C, C // groups)))
              and kind in ("silu", "sigmoid"), "gated_groupnorm: bad operands")
        out = torch.empty(T, C, dtype=out_dtype, device=y.device)
        gp, gs = self._rows_f32(gate, "gated_groupnorm gate")
        _check(self.lib.ifx_gated_groupnorm(y, gp, gs, w, 0 if w is None else int(w.numel()), float(eps), out, T, C,
                                            int(groups), int(bool(gate_first)), int(kind == "sigmoid"), _DT[out_dtype], _stream()),
               "gated_groupnorm")
        self.launches += 1
        return out

    def pair_combine(self, a, b, w_a, w_b, c_a, c_b, eps):
        """float32 [T, C]: c_a a + c_b b, or with weights c_a a / rms(a) * w_a + c_b b / rms(b) * w_b (a, b in any dtype)."""
        T, C = a.shape
        _need(a.is_contiguous() and b.is_contiguous() and a.shape == b.shape and (w_a is None) == (w_b is None),
              "pair_combine: rows of one shape")
        out = torch.empty(T, C, dtype=torch.float32, device=a.device)
        _check(self.lib.ifx_pair_combine(a, _DT[a.dtype], b, _DT[b.dtype], w_a, w_b, float(c_a),
                                         float(c_b), float(eps), out, T, C, _stream()), "pair_combine")
        self.launches += 1
        return out

    def residual_add_vectors(self, x, a, s_a, b=None, s_b=None, b2=None):
        """x += s_a * a + s_b * (b + b2), element by element along a row (a vector None: ones; b, b2 may be None)."""
        T, C = x.shape
        a = self.materialize(a)
        b = None if b is None else self.materialize(b)
        b2 = None if b2 is None else self.materialize(b2)
        if b is not None and b2 is not None and b2.dtype != b.dtype:
            b2 = b2.to(b.dtype)
        _need(x.dtype == torch.float32 and x.is_contiguous() and a.shape == x.shape and a.is_contiguous()
              and (b is None or (b.shape == x.shape and b.is_contiguous())) and (b2 is None or (b is not None and b2.is_contiguous())),
              "residual_add_vectors: bad operands")
        _check(self.lib.ifx_residual_add_vectors(x, a, _DT[a.dtype], s_a, b, b2,
                                                 _DT[b.dtype] if b is not None else 0, s_b, T, C, _stream()),
               "residual_add_vectors")
        self.launches += 1

    # ------------------------------------------- norms of sums, rotated rows, an elementwise recurrence
    def norm_of_sum(self, x, alpha, terms, w, eps, out_dtype=None):
        """x <- n(alpha x + sum c (y + bias)), float32 and in place, for one or two terms (c, y, bias): y a tensor or a
        PartialSum, bias float32 along the row or None; n the RMS norm times w (w None: x is the sum itself).  With
        `out_dtype` also returns the new rows in that dtype."""
        T, H = x.shape
        _need(x.dtype == torch.float32 and x.is_contiguous() and 1 <= len(terms) <= 2
              and (w is None or (w.dtype == torch.float32 and w.numel() == H and w.is_contiguous())), "norm_of_sum: bad operands")
        flat = []
        for c, y, bias in list(terms) + [(0.0, None, None)] * (2 - len(terms)):
            splits = 1
            if isinstance(y, PartialSum):
                _need(tuple(y.shape) == (T, H), "norm_of_sum: partial sums do not match x")
                y, splits = y.parts, y.splits
            _need((y is None or (tuple(y.shape[-2:]) == (T, H) and y.is_contiguous()))
                  and (bias is None or (bias.dtype == torch.float32 and bias.numel() == H and bias.is_contiguous())),
                  "norm_of_sum: a term does not match x")
            flat += [y, 0 if y is None else _DT[y.dtype], splits, float(c), bias]
        out = None if out_dtype is None else torch.empty(T, H, dtype=out_dtype, device=x.device)
        _check(self.lib.ifx_norm_of_sum(x, float(alpha), *flat, w, float(eps), out,
                                        0 if out is None else _DT[out_dtype], T, H, _stream()), "norm_of_sum")
        self.launches += 1
        return out

    def joins_projections(self, h):
        """Whether two stacked projections of the same rows run as one product: for few bfloat16 rows, where the time is the
        weights' way in; with many rows each keeps an output dtype of its own."""
        return h.dtype == torch.bfloat16 and h.shape[0] <= self.SKINNY_MAX_ROWS

    @staticmethod
    def _row_source(rows):
        """(plain pointer, dtype code, partial pointer, splits, row length) of a tensor or PartialSum."""
        if isinstance(rows, PartialSum):
            return None, 0, rows.parts, rows.splits, rows.parts.shape[-1]
        _need(rows.is_contiguous(), "projected rows must be contiguous")
        return rows, _DT[rows.dtype], None, 1, rows.shape[-1]

    def row_norm_rope_append(self, rows, col0, bias, rotary, turn, temp, nq, nkv, d, dv, ctx, cache, q_norm=None, k_norm=None,
                             norm_eps=0.0, v_from_k=False, gate_col=None):
        """Columns col0 .. of `rows` (a tensor or PartialSum): [nq heads of d | nkv key heads of d | nkv value heads of dv],
        plus `bias`; the query part and the key part RMS-normed as a whole (weights of their full size; None: no norm),
        turned by `rotary`, the queries times `temp` per head; the values turned by `turn` over their whole heads; keys and
        values to the cache.  Returns (queries [T, nq d] in the cache's dtype, what `attention` takes as `turn_back`).
        `v_from_k`: no value columns, the values are the keys with their bias, in front of norm and rotation.  With `gate_col`
        returns a third: sigmoid of the nq columns from col0 + gate_col on, float32 [T, nq] (no bias)."""
        T = rows.shape[0]
        kv, table = cache.kv, cache.block_table
        _need(kv is not None and table is not None and kv.shape[1] == 2 and kv.shape[2] == nkv and kv.shape[-1] >= max(d, dv),
              "row_norm_rope_append: the cache does not fit the heads")
        _need(not v_from_k or dv == d, "row_norm_rope_append: values that are the keys have their size")
        for v, n in ((bias, nq * d + nkv * (d if v_from_k else d + dv)), (q_norm, nq * d), (k_norm, nkv * d), (temp, nq)):
            _need(v is None or (v.dtype == torch.float32 and v.numel() == n and v.is_contiguous()),
                  "row_norm_rope_append: biases, norm weights and factors are float32 of their full size")
        for table_, size in ((rotary, d), (turn, dv)):
            _need(table_ is None or (table_.magnitude == 1.0 and table_.rotary_dim <= size), "row_norm_rope_append: a table does not fit")
        _need(turn is None or turn.rotary_dim == dv, "row_norm_rope_append: values are turned as a whole")
        src, code, part, splits, ld = self._row_source(rows)
        dev = kv.device
        q_out = torch.empty(T, nq * d, dtype=kv.dtype, device=dev)
        back = None if turn is None else torch.empty(T, dv // 2, 2, dtype=torch.float32, device=dev)
        gate = None if gate_col is None else torch.empty(T, nq, dtype=torch.float32, device=dev)
        _check(self.lib.ifx_row_norm_rope_append(
            src, code, part, splits, ld, int(col0), bias, q_norm, k_norm, float(norm_eps),
            (None if rotary is None else rotary.inv_freq), 0 if rotary is None else int(rotary.rotary_dim),
            int(rotary is not None and rotary.interleaved), (None if turn is None else turn.inv_freq),
            int(turn is not None and turn.interleaved), temp, ctx.positions, ctx.token_req, ctx.req_slot,
            table, table.shape[1], cache.page_size, kv.shape[0], kv, q_out, back, T, nq, nkv, d, dv,
            kv.shape[-1], int(bool(cache.writes)), int(bool(v_from_k)), gate, int(gate_col or 0), _DT[kv.dtype], _stream()),
            "row_norm_rope_append")
        self.launches += 1
        turned = None if back is None else (back, turn.interleaved)
        return (q_out, turned) if gate_col is None else (q_out, turned, gate)

    def silu_columns(self, rows, acted, ctx):
        """float32 rows from `rows` (a float32 tensor, changed in place, or a PartialSum): z sigmoid(z) on the first `acted`
        columns, the others as they are."""
        T = rows.shape[0]
        src, code, part, splits, ld = self._row_source(rows)
        plain = not isinstance(rows, PartialSum)
        _need(not plain or rows.dtype == torch.float32, "silu_columns: float32 rows")
        out = rows if plain else torch.empty(T, ld, dtype=torch.float32, device=rows.parts.device)
        _check(self.lib.ifx_silu_columns(src, part, splits, ld, 0, out, T, int(ld), int(acted), _stream()), "silu_columns")
        self.launches += 1
        return out

    def rotate_rows(self, rows, col0, width, heads, dk, rotary, k_scale, ctx):
        """float32 [T, width] from columns col0 .. of `rows` (a float32 tensor, which is then changed in place where it has
        just these columns, or a PartialSum): heads of dk (queries), heads of dk (keys), the rest; queries and keys turned
        by the position, keys times k_scale behind it."""
        T = rows.shape[0]
        src, code, part, splits, ld = self._row_source(rows)
        plain = not isinstance(rows, PartialSum)
        _need(not plain or rows.dtype == torch.float32, "rotate_rows: float32 rows")
        _need(rotary is None or (rotary.magnitude == 1.0 and rotary.rotary_dim <= dk), "rotate_rows: the table does not fit")
        device = rows.device if plain else rows.parts.device
        out = rows if plain and ld == width and col0 == 0 else torch.empty(T, width, dtype=torch.float32, device=device)
        _check(self.lib.ifx_rotate_rows(
            src, part, splits, ld, int(col0), (None if rotary is None else rotary.inv_freq),
            0 if rotary is None else int(rotary.rotary_dim), int(rotary is not None and rotary.interleaved), ctx.positions,
            out, T, int(width), int(heads), int(dk), float(k_scale), _stream()), "rotate_rows")
        self.launches += 1
        return out

    def gated_scan(self, rows, bias, state, width, ctx, out_dtype):
        """rows [T, 3 width] (float32 or PartialSum) = z, x, g; `bias` (float32 [2 width]) joins z and x:
        S <- (1 - sigmoid(z)) S + sigmoid(z) c with c = x + 1/2 where x >= 0 and sigmoid(x) where x < 0; returns S silu(g) in
        `out_dtype`.  S per request in `state` (float32 [slots, >= width]), moved on."""
        T = rows.shape[0]
        _need(tuple(rows.shape) == (T, 3 * width) and bias.dtype == torch.float32 and bias.numel() == 2 * width
              and state is not None and state.dtype == torch.float32 and state.stride(1) == 1 and state.shape[1] >= width,
              "gated_scan: bad operands")
        src, splits = (rows.parts, rows.splits) if isinstance(rows, PartialSum) else (rows, 1)
        _need(src.dtype == torch.float32 and src.is_contiguous(), "gated_scan: float32 rows")
        out = torch.empty(T, width, dtype=out_dtype, device=src.device)
        _check(self.lib.ifx_gated_scan(src, splits, bias, state, state.stride(0), ctx.req_slot,
                                       ctx.cu_seqlens, out, ctx.num_requests, T, int(ctx.max_span), int(width),
                                       _DT[out_dtype], _stream()), "gated_scan")
        self.launches += 1
        return out

    # ---------------------------------------------------------------- sampling
    def argmax(self, logits):
        R, V = logits.shape
        out = torch.empty(R, dtype=torch.int32, device=logits.device)
        if V >= 16384 and R <= 256:                      # long rows, few of them: many blocks per row
            _check(self.lib.ifx_argmax_chunks(logits, out, R, V, 32, self._argmax_val,
                                              self._argmax_idx, self._argmax_tickets, _stream()), "argmax")
            self.launches += 1
            return out
        _check(self.lib.ifx_argmax(logits, out, R, V, _stream()), "argmax")
        self.launches += 1
        return out

    def penalties(self, logits, tokens, counts, rep, freq, pres):
        R, V = logits.shape
        _check(self.lib.ifx_penalties(logits, tokens, counts, rep, freq, pres,
                                      R, tokens.shape[1], V, _stream()), "penalties")
        self.launches += 1

    def logit_bias(self, logits, rows, tokens, bias):
        R, V = logits.shape
        _check(self.lib.ifx_logit_bias(logits, rows, tokens, bias, rows.numel(), R, V,
                                       _stream()), "logit_bias")
        self.launches += 1

    def sample(self, logits, temperature, top_k, top_p, min_p, seed_lo, seed_hi, step, features=3):
        """One draw per row (see sampling.cu).  Rows are spread over many blocks; `features` says which
        filters any row uses (bit 0: top-k, bit 1: top-p) so that the passes of the others are not launched."""
        R, V = logits.shape
        out = torch.empty(R, dtype=torch.int32, device=logits.device)
        if R > self._sample_capacity:                    # the scratch's layout goes with its capacity
            self._sample_capacity = max(64, 1 << (R - 1).bit_length())
            self._sample_scratch = torch.zeros(int(self.lib.ifx_sample_scratch_bytes(self._sample_capacity)),
                                               dtype=torch.uint8, device=logits.device)
        passes = 3 + (1 if features & 3 else 0) + (2 if features & 1 else 0) + (3 if features & 2 else 0)
        _check(self.lib.ifx_sample_blocks(logits, temperature, top_k, top_p, min_p,
                                          seed_lo, seed_hi, step, out, R, V, int(features),
                                          self._sample_scratch, self._sample_capacity, _stream()), "sample")
        self.launches += passes
        return out

    def sample_one_block(self, logits, temperature, top_k, top_p, min_p, seed_lo, seed_hi, step):
        """The same draw with one block per row and thresholds by bisection (kept for comparison)."""
        R, V = logits.shape
        probs = torch.empty(R, V, dtype=torch.float32, device=logits.device)
        out = torch.empty(R, dtype=torch.int32, device=logits.device)
        _check(self.lib.ifx_sample(logits, probs, temperature, top_k, top_p,
                                   min_p, seed_lo, seed_hi, step, out, R, V,
                                   _stream()), "sample")
        self.launches += 1
        return out
