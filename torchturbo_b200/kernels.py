"""Bindings for the sm_100a CUDA library (`_lib/libttb200.so`): ctypes, and for the operators that a training step calls by the
hundred the extension module `_lib/ttb_host.so` (csrc/host.cpp).

Every function here launches hand-written kernels on the *current* CUDA stream
and takes/returns torch tensors.  Nothing falls back to PyTorch: if the library
is missing on a machine with a GPU, `lib()` raises so that a silent eager path
can never pass for the native one.  CPU-only processes never touch this module
(the op dispatcher selects the torch providers there).
"""
from __future__ import annotations

import ctypes as C
import importlib.machinery
import importlib.util
from functools import lru_cache
from pathlib import Path

import torch

_LIB_PATH = Path(__file__).resolve().parent / "_lib" / "libttb200.so"
_HOST_PATH = _LIB_PATH.with_name("ttb_host.so")
_lib = None
_host = None

SEG_ALIGN = 128  # rows; every expert segment of a permuted buffer is padded to this
SCORE_FN = {"softmax_pre": 0, "softmax_post": 1, "sigmoid": 2}


class KernelError(RuntimeError):
    pass


class EpFuseArgs(C.Structure):
    """Expert-parallel fusion of one grouped GEMM launch (`struct EpFuseArgs` of csrc/gemm.cu): the push prologue that
    sends this rank's routed rows to their owners from inside the kernel, and / or the scatter epilogue that stores every
    output row into the return buffer of the rank it came from."""

    _fields_ = [
        ("peer_ptrs", C.c_void_p), ("W", C.c_int), ("rank", C.c_int), ("El", C.c_int),
        ("status", C.c_void_p), ("budget_ms", C.c_longlong),
        ("push_on", C.c_int),
        ("off_rows", C.c_longlong), ("off_vals", C.c_longlong), ("off_tags", C.c_longlong), ("off_flags", C.c_longlong),
        ("src", C.c_void_p), ("lds", C.c_longlong),
        ("order", C.c_void_p), ("expert", C.c_void_p), ("dest_row", C.c_void_p), ("val", C.c_void_p),
        ("counts", C.c_void_p), ("sent", C.c_void_p),
        ("n_entries", C.c_int), ("k", C.c_int), ("H", C.c_int), ("epoch", C.c_int),
        ("cap_rows", C.c_longlong),
        ("scat_on", C.c_int),
        ("off_ret", C.c_longlong), ("off_ret_vals", C.c_longlong), ("off_ret_flags", C.c_longlong),
        ("row_tag", C.c_void_p), ("row_val", C.c_void_p),
        ("ret_epoch", C.c_int),
        ("done_counter", C.c_void_p),
        ("ret_rows", C.c_int),
    ]


def lib_path() -> Path:
    return _LIB_PATH


def is_built() -> bool:
    return _LIB_PATH.exists()


def available() -> bool:
    """True when the CUDA library can be used in this process."""
    return torch.cuda.is_available() and is_built()


def lib():
    global _lib
    if _lib is None:
        if not _LIB_PATH.exists():
            raise KernelError(
                f"{_LIB_PATH} is missing: run `python -m torchturbo_b200.csrc.build` "
                "(or __graft_entry__.build()) before using the CUDA ops"
            )
        _lib = C.CDLL(str(_LIB_PATH))
    return _lib


def host():
    """The launch functions of the hot operators."""
    global _host
    if _host is None:
        lib()
        if not _HOST_PATH.exists():
            raise KernelError(f"{_HOST_PATH} is missing: run `python -m torchturbo_b200.csrc.build` (or __graft_entry__.build())")
        loader = importlib.machinery.ExtensionFileLoader("ttb_host", str(_HOST_PATH))
        module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("ttb_host", str(_HOST_PATH), loader=loader))
        loader.exec_module(module)
        module.setup(KernelError, torch.OutOfMemoryError, gemm_splits)
        _host = module
    return _host


# kernels launched per C entry point (used to report how many of this library's kernels ran in a region)
_LAUNCHES_PER_CALL = {"ttb_gated_rmsnorm_bwd": 2, "ttb_causal_conv1d_bwd": 2,
                      "ttb_causal_conv1d_row_blocks": 0, "ttb_ep_dispatch_all": 5, "ttb_ep_dispatch_rows": 3,
                      "ttb_ep_combine_all": 3, "ttb_delta_vec_bwd_post": 2, "ttb_ep_combine_vals": 4, "ttb_ep_prepare": 3, "ttb_ep_prepare_bwd": 1, "ttb_router_fwd": 2, "ttb_perm_index": 3, "ttb_perm_scatter": 2,
                      "ttb_gemm_status": 0}
LAUNCH_COUNT = 0


def launch_count() -> int:
    """Number of CUDA kernels of this library launched so far in this process."""
    return LAUNCH_COUNT + (_host.launches() if _host is not None else 0)


def _check(code: int, what: str) -> None:
    global LAUNCH_COUNT
    if code != 0:
        raise KernelError(f"{what} failed with code {code}")
    LAUNCH_COUNT += _LAUNCHES_PER_CALL.get(what, 1)


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream() -> C.c_void_p:
    """Handle of the current stream of the current device (the raw accessor skips building a `torch.cuda.Stream`)."""
    if _raw_stream is not None:
        return C.c_void_p(_raw_stream(torch.cuda.current_device()))
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def check_device(t: torch.Tensor) -> None:
    """Kernels run on the current device's stream: an operand of another GPU would be an illegal address there."""
    if t.device.index != torch.cuda.current_device():
        raise KernelError(f"operand lives on {t.device} but the current CUDA device is {torch.cuda.current_device()}; "
                          "call torch.cuda.set_device() for this process before using the ops")


def _p(t: torch.Tensor | None) -> C.c_void_p:
    return C.c_void_p(0 if t is None else t.data_ptr())


@lru_cache(maxsize=None)
def num_sms(device_index: int | None = None) -> int:
    return torch.cuda.get_device_properties(device_index if device_index is not None else torch.cuda.current_device()).multi_processor_count


def status(reset: bool = False) -> tuple[int, int]:
    """(first error code, number of errors) recorded by bounded in-kernel waits of the GEMM unit."""
    buf = (C.c_uint * 4)()
    _check(lib().ttb_gemm_status(buf, C.c_int(1 if reset else 0)), "ttb_gemm_status")
    return int(buf[0]), int(buf[1])


# --------------------------------------------------------------------------------------
# GEMM
# --------------------------------------------------------------------------------------
def gemm_splits(M: int, N: int, K: int, sms: int) -> int:
    """Into how many pieces along K a dense product is cut.  A product with few output tiles keeps few SMs busy for
    ``K / 64`` steps each; cut in ``S`` pieces it keeps ``S`` times as many busy for ``1 / S`` of the steps, plus a pass over
    ``S`` fp32 partial results.  Worth it while at most half of the SMs have a tile and a piece keeps 32 k-blocks (the pieces
    are equal but for the last, which takes what is left: 97 blocks go 33, 33, 31), so that the loop outweighs the second
    launch (6 tiles of 500 steps, the input gradient of a 32000-row loss head: 150 us less for a sum of 4 us); short K stays
    whole."""
    tiles = ((M + 127) // 128) * ((N + 255) // 256 if N > 128 else 1)
    if N % 8 or tiles == 0:
        return 1
    return max(1, min(sms // tiles, (K + 63) // 64 // 32))


def _is_f32(dtype: torch.dtype) -> bool:
    assert dtype in (torch.bfloat16, torch.float32), dtype
    return dtype == torch.float32


def gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    *,
    a_mn: bool = False,
    b_mn: bool = False,
    out: torch.Tensor | None = None,
    out_dtype: torch.dtype = torch.bfloat16,
    accumulate: bool = False,
    residual: torch.Tensor | None = None,
    tile_group: torch.Tensor | None = None,
    group_rows: torch.Tensor | None = None,
    swiglu: bool = False,
    row_scale: torch.Tensor | None = None,
    preact: torch.Tensor | None = None,
    ep: "EpFuseArgs | None" = None,
    alpha: torch.Tensor | None = None,
) -> torch.Tensor:
    """tcgen05 GEMM ``C = op(A) @ op(B)`` on bf16 operands with fp32 accumulation.

    Memory orientation (row-major tensors):
      * ``a_mn=False``: ``a`` is ``[M, K]``;  ``a_mn=True``: ``a`` is ``[K, M]`` (used as its transpose).
      * ``b_mn=False``: ``b`` is ``[N, K]`` (``nn.Linear`` weight); ``b_mn=True``: ``b`` is ``[K, N]``.
      * grouped-M (``tile_group`` given): ``b`` is ``[G, N, K]`` / ``[G, K, N]`` and 128-row tile ``i`` of
        ``a`` multiplies ``b[tile_group[i]]`` (negative = skip the tile).
      * grouped-K (``group_rows`` given, both operands MN-major): ``C[g] = a[r_g:r_{g+1}].T @ b[r_g:r_{g+1}]``
        with ``group_rows`` an int32 ``[G+1]`` device tensor of 64-aligned row offsets.
      * ``swiglu=True``: ``b`` holds ``[gate | up]`` output columns (``2F``); the result is
        ``silu(gate) * up * row_scale`` of width ``F``; ``preact`` (``[M, 2F]``) optionally keeps gate|up.
      * ``alpha`` (one fp32 value on the device) is multiplied into the fp32 product before it is rounded or added.
    """
    return host().gemm(a, b, a_mn, b_mn, out, _is_f32(out_dtype), accumulate, residual, tile_group, group_rows, swiglu, row_scale, preact,
                       C.addressof(ep) if ep is not None else 0, alpha)


# --------------------------------------------------------------------------------------
# RMSNorm
# --------------------------------------------------------------------------------------
def rmsnorm_fwd(x, weight, eps, residual=None, one_plus_w=False):
    """Returns (y, rstd, x_sum) where x_sum is ``x + residual`` (or ``x`` itself without residual)."""
    return host().rmsnorm_fwd(x, weight, eps, residual, one_plus_w)


def rmsnorm_bwd(dy, x_sum, weight, rstd, dres=None, one_plus_w=False, dw_dtype=torch.float32):
    """Returns (dx, dw in ``dw_dtype``: fp32 or bf16); ``dres`` (gradient arriving on the residual stream) is added into dx."""
    return host().rmsnorm_bwd(dy, x_sum, weight, rstd, dres, one_plus_w, dw_dtype != torch.bfloat16)


def _gated_grid(R: int, H: int, device) -> int:
    rows = 2048 // H                       # rows of one 256-thread block
    return max(1, min((R + rows - 1) // rows, 8 * num_sms(device.index)))


def gated_rmsnorm_fwd(x, gate, weight, eps, silu: bool):
    """``bf16(rmsnorm(x) * weight) * act(gate)`` on bf16 rows of 64, 128 or 256 channels.  Returns (y, rstd)."""
    R, H = x.shape
    y = torch.empty_like(x)
    rstd = torch.empty(R, dtype=torch.float32, device=x.device)
    _check(lib().ttb_gated_rmsnorm_fwd(_p(x), _p(gate), _p(weight), _p(y), _p(rstd), C.c_longlong(R), C.c_int(H), C.c_float(eps),
                                       C.c_int(int(silu)), C.c_int(_gated_grid(R, H, x.device)), _stream()), "ttb_gated_rmsnorm_fwd")
    return y, rstd


def gated_rmsnorm_bwd(dy, x, gate, weight, rstd, silu: bool):
    """Returns (dx, dgate, dw), all bf16."""
    R, H = x.shape
    grid = _gated_grid(R, H, x.device)
    dx, dgate = torch.empty_like(x), torch.empty_like(x)
    dw = torch.empty_like(weight) if R else torch.zeros_like(weight)
    partial = torch.empty(grid, H, dtype=torch.float32, device=x.device)
    _check(lib().ttb_gated_rmsnorm_bwd(_p(dy), _p(x), _p(gate), _p(weight), _p(rstd), _p(dx), _p(dgate), _p(partial), _p(dw),
                                       C.c_longlong(R), C.c_int(H), C.c_int(int(silu)), C.c_int(grid), _stream()),
           "ttb_gated_rmsnorm_bwd")
    return dx, dgate, dw


# --------------------------------------------------------------------------------------
# LayerNorm and bias + activation (vision tower)
# --------------------------------------------------------------------------------------
ACT = {None: 0, "none": 0, "identity": 0, "gelu_tanh": 1, "gelu_pytorch_tanh": 1, "gelu": 2, "gelu_erf": 2}


def layernorm_fwd(x, weight, bias, eps):
    """Returns (y, mean, rstd); statistics in fp32."""
    return host().layernorm_fwd(x, weight, bias, eps)


def layernorm_bwd(dy, x, weight, mean, rstd, dw_dtype=torch.float32):
    """Returns (dx, dw, db), the last two in ``dw_dtype`` (fp32 or bf16)."""
    return host().layernorm_bwd(dy, x, weight, mean, rstd, dw_dtype != torch.bfloat16)


def bias_act_fwd(x, bias, act, residual=None):
    """y = act(x + bias) (+ residual) on bf16 rows."""
    return host().bias_act_fwd(x, bias, ACT[act], residual)


def bias_act_bwd(dy, x, bias, act, db_dtype=torch.float32):
    """Returns (dx, dbias in ``db_dtype``: fp32 or bf16); with the identity activation dx is dy itself."""
    return host().bias_act_bwd(dy, x, bias, ACT[act], db_dtype != torch.bfloat16)


# --------------------------------------------------------------------------------------
# causal depthwise short convolution (linear-attention mixers)
# --------------------------------------------------------------------------------------
def causal_conv1d_fwd(x, weight, bias, seq_start, silu: bool):
    """x [T, D] bf16, weight [D, W] bf16, seq_start int32 [T] (first token of each token's sequence) -> y [T, D]."""
    T, D = x.shape
    y = torch.empty_like(x)
    _check(lib().ttb_causal_conv1d_fwd(_p(x), _p(weight), _p(bias), _p(seq_start), _p(y), C.c_longlong(T), C.c_int(D),
                                       C.c_int(weight.shape[1]), C.c_int(int(silu)), _stream()), "ttb_causal_conv1d_fwd")
    return y


def causal_conv1d_bwd(dy, x, weight, bias, seq_start, seq_end, silu: bool):
    """Returns (dx [T, D] bf16, dw [D, W] fp32, db [D] fp32)."""
    T, D = x.shape
    W = weight.shape[1]
    blocks = int(lib().ttb_causal_conv1d_row_blocks(C.c_longlong(T), C.c_int(D), C.c_int(W)))
    dpre = torch.empty_like(x) if W > 4 else None       # shorter filters form dx in the same pass
    dx = torch.empty_like(x)
    part = torch.empty(blocks, (W + 1) * D, dtype=torch.float32, device=x.device)
    dwdb = torch.empty(W + 1, D, dtype=torch.float32, device=x.device)
    _check(lib().ttb_causal_conv1d_bwd(_p(dy), _p(x), _p(weight), _p(bias), _p(seq_start), _p(seq_end), _p(dpre), _p(dx),
                                       _p(part), _p(dwdb), C.c_longlong(T), C.c_int(D), C.c_int(W), C.c_int(int(silu)),
                                       _stream()), "ttb_causal_conv1d_bwd")
    global LAUNCH_COUNT
    LAUNCH_COUNT += 1 if W > 4 else 0
    # plane s holds the tap at distance s into the past = weight column W-1-s
    dw = dwdb[:W].flip(0).t().contiguous()
    return dx, dw, dwdb[W]


# --------------------------------------------------------------------------------------
# QK-norm + RoPE
# --------------------------------------------------------------------------------------
def qknorm_rope_fwd(qkv, n_q, n_kv, head_dim, wq, wk, cos, sin, eps, use_norm=True):
    """qkv: [T, (n_q + 2 n_kv) * D] -> (q [T, n_q, D], k [T, n_kv, D], rstd [T * (n_q + n_kv)])."""
    return host().qknorm_rope_fwd(qkv, n_q, n_kv, head_dim, wq, wk, cos, sin, eps, use_norm)


def qknorm_rope_bwd(dq, dk, qkv, n_q, n_kv, head_dim, wq, wk, cos, sin, rstd, dqkv, use_norm=True, dv=None, dw_dtype=torch.float32):
    """Writes the q and k column blocks of ``dqkv`` ([T, ld]), with ``dv`` ([T, n_kv, D]) the v block too, and returns (dwq, dwk)
    in ``dw_dtype`` (fp32 or bf16)."""
    return host().qknorm_rope_bwd(dq, dk, dv, qkv, n_q, n_kv, head_dim, wq, wk, cos, sin, rstd, dqkv, use_norm, dw_dtype != torch.bfloat16)


def qkv_rope_fwd(x, bias, heads, cos, sin):
    """x: [T, 3 * heads * D] -> q, k = RoPE(x + bias), v = x + bias, each [T, heads, D]; cos, sin fp32 [T, D / 2]."""
    return host().qkv_rope_fwd(x, bias, heads, cos, sin)


def qkv_rope_bwd(dq, dk, dv, cos, sin, db_dtype=torch.float32):
    """Returns (dx [T, 3 * heads * D], dbias in ``db_dtype``: fp32 or bf16)."""
    return host().qkv_rope_bwd(dq, dk, dv, cos, sin, db_dtype != torch.bfloat16)


def rope(x, cos, sin, sign: float = 1.0):
    """Half-rotation RoPE of bf16 [T, heads, D] (channels contiguous); cos, sin fp32 [T, D / 2].  ``sign=-1`` rotates back."""
    return host().rope(x, cos, sin, sign)


# --------------------------------------------------------------------------------------
# Kimi delta attention gate
# --------------------------------------------------------------------------------------
def kda_gate_fwd(g, A_log, dt_bias, lower_bound):
    """Log decay fp32 [rows, H, 128] from the bf16 projection `g`; A_log [H] and dt_bias [H * 128] (or None) in bf16 or fp32."""
    return host().kda_gate_fwd(g, A_log, dt_bias, lower_bound is not None, lower_bound or 0.0)


def kda_gate_bwd(dd, g, A_log, dt_bias, lower_bound):
    """(dg bf16, d(dt) fp32 [H * 128], channel sums of d(A_log) fp32 [H, 128])."""
    return host().kda_gate_bwd(dd, g, A_log, dt_bias, lower_bound is not None, lower_bound or 0.0)


def gdn_gate_fwd(a, b, A_log, dt_bias):
    """(g = -exp(A_log) softplus(a + dt_bias), beta = sigmoid(b)), fp32 [T, H], of bf16 projections [T, H]."""
    return host().gdn_gate_fwd(a, b, A_log, dt_bias)


def gdn_gate_bwd(dg, dbeta, a, A_log, dt_bias, beta, dtype=torch.float32):
    """(da, db bf16, d(A_log), d(dt_bias) in ``dtype``: fp32 or bf16)."""
    return host().gdn_gate_bwd(dg, dbeta, a, A_log, dt_bias, beta, dtype != torch.bfloat16)


# --------------------------------------------------------------------------------------
# SwiGLU
# --------------------------------------------------------------------------------------
def swiglu_fwd(x, row_scale=None, nrows=None):
    """`nrows` (int32 device scalar, optional): only the first `nrows[0]` rows are computed (padded buffers)."""
    return host().swiglu_fwd(x, row_scale, nrows)


def swiglu_bwd(dy, x, row_scale=None, want_dscale=False, nrows=None, y_out=None):
    """`nrows` (int32 device scalar, optional): rows from `nrows[0]` on are left untouched (padded buffers).  `y_out` (bf16
    [R, F], optional) receives the forward result, as `swiglu_fwd` computes it."""
    return host().swiglu_bwd(dy, x, row_scale, want_dscale, nrows, y_out)


# --------------------------------------------------------------------------------------
# Cross entropy
# --------------------------------------------------------------------------------------
def cross_entropy(logits, labels, *, grad_out=None, grad_scale=None, grad_scale_host=1.0, want_lse=False):
    """Per-row CE (fp32, 0 for ignored rows).  With ``grad_out`` (bf16 [R, V]; may alias bf16 logits) also writes
    ``(softmax - onehot) * grad_scale[0] * grad_scale_host``."""
    R, V = logits.shape
    assert labels.dtype == torch.int64 and labels.numel() == R
    loss = torch.empty(R, dtype=torch.float32, device=logits.device)
    lse = torch.empty(R, dtype=torch.float32, device=logits.device) if want_lse else None
    _check(lib().ttb_cross_entropy(_p(logits), C.c_int(int(logits.dtype == torch.float32)),
                                   C.c_longlong(logits.stride(0)), _p(labels), _p(loss), _p(lse), _p(grad_out),
                                   C.c_longlong(grad_out.stride(0) if grad_out is not None else 0), _p(grad_scale),
                                   C.c_float(grad_scale_host), C.c_longlong(R), C.c_int(V), _stream()),
           "ttb_cross_entropy")
    return (loss, lse) if want_lse else loss


# --------------------------------------------------------------------------------------
# Multi-tensor AdamW / grad norm
# --------------------------------------------------------------------------------------
ADAM_CHUNK = 16384


def copy_words(dst: torch.Tensor, src: torch.Tensor) -> None:
    """Copy between the device and pinned host memory on the current stream: contiguous tensors of one type, whole 32-bit words."""
    host().copy_words(dst, src)


class MultiTensorPlan:
    """Device tables for the multi-tensor AdamW / squared-norm kernels.

    ``meta`` rows are ``(p, g, m, v, shadow, numel, g_is_bf16)`` as int64; the chunk table maps each CUDA block to
    ``(tensor index, chunk index)``.  Gradient pointers are refreshed every step (autograd reallocates them).
    """

    def __init__(self, params, exp_avg, exp_avg_sq, shadows=None):
        self.params = list(params)
        self.device = self.params[0].device
        n = len(self.params)
        self.host_meta = torch.zeros(n, 7, dtype=torch.int64).pin_memory()
        assert all(p.dtype == torch.float32 and p.is_contiguous() for p in self.params)
        rows = self.host_meta.numpy()
        rows[:, 0] = [p.data_ptr() for p in self.params]
        rows[:, 2] = [t.data_ptr() for t in exp_avg[:n]]
        rows[:, 3] = [t.data_ptr() for t in exp_avg_sq[:n]]
        rows[:, 4] = [t.data_ptr() if t is not None else 0 for t in (shadows[:n] if shadows is not None else [None] * n)]
        rows[:, 5] = [p.numel() for p in self.params]
        counts = (self.host_meta[:, 5] + ADAM_CHUNK - 1) // ADAM_CHUNK
        self.n_chunks = int(counts.sum())
        tensor = torch.repeat_interleave(torch.arange(n), counts)
        chunk = torch.arange(self.n_chunks) - torch.repeat_interleave(counts.cumsum(0) - counts, counts)
        self.chunks = torch.stack((tensor, chunk), 1).to(torch.int32).contiguous().to(self.device)
        self.meta = torch.empty(n, 7, dtype=torch.int64, device=self.device)
        self.partial = torch.empty(max(self.n_chunks, 1), dtype=torch.float32, device=self.device)

    def refresh_grads(self, grads):
        # the pinned table is read by the previous refresh's asynchronous copy until that copy has run on the device:
        # a host that is a whole step ahead waits here instead of overwriting pointers still to be copied
        ev = getattr(self, "_copy_event", None)
        if ev is not None:
            ev.synchronize()
        # the table through a numpy view: an element assignment to a tensor costs microseconds, and there are two per gradient
        rows = self.host_meta.numpy()
        assert rows[:, 5].tolist() == [g.numel() for g in grads] and all(g.is_contiguous() for g in grads)
        rows[:, 1] = [g.data_ptr() for g in grads]
        rows[:, 6] = [g.dtype == torch.bfloat16 for g in grads]
        if self.device.type != "cuda":
            self.meta.copy_(self.host_meta)
        else:
            copy_words(self.meta, self.host_meta)
            self._copy_event = torch.cuda.Event()
            self._copy_event.record()


def grad_sqnorm_partials(plan: MultiTensorPlan, prescale: float = 1.0) -> torch.Tensor:
    _check(lib().ttb_grad_sqnorm(_p(plan.meta), _p(plan.chunks), C.c_int(plan.n_chunks), _p(plan.partial),
                                 C.c_float(prescale), _stream()), "ttb_grad_sqnorm")
    return plan.partial[: plan.n_chunks]


def clip_coef(partials: torch.Tensor, max_norm: float, extra_sq: torch.Tensor | None = None) -> torch.Tensor:
    """Returns a device tensor ``[sum_sq, norm, coef]`` with ``coef = min(1, max_norm / (norm + 1e-6))``."""
    out = torch.empty(3, dtype=torch.float32, device=partials.device)
    _check(lib().ttb_clip_coef(_p(partials), C.c_int(partials.numel()), _p(extra_sq), C.c_float(max_norm), _p(out),
                               _stream()), "ttb_clip_coef")
    return out


def adamw_step(plan: MultiTensorPlan, *, lr, beta1, beta2, eps, weight_decay, step, clip=None, grad_prescale=1.0):
    bc1 = 1.0 - beta1 ** step
    bc2_sqrt = (1.0 - beta2 ** step) ** 0.5
    _check(lib().ttb_adamw(_p(plan.meta), _p(plan.chunks), C.c_int(plan.n_chunks), C.c_float(lr), C.c_float(beta1),
                           C.c_float(beta2), C.c_float(eps), C.c_float(weight_decay), C.c_float(bc1),
                           C.c_float(bc2_sqrt), _p(clip), C.c_float(grad_prescale), _stream()), "ttb_adamw")


def scale(x: torch.Tensor, factor: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """`(x.float() * factor).to(dtype)` in one pass: x contiguous bf16 or fp32, factor one fp32 value on the device, dtype bf16 or fp32."""
    assert dtype in (torch.bfloat16, torch.float32)
    return host().scale(x, factor, dtype == torch.bfloat16)


# --------------------------------------------------------------------------------------
# MoE router / permutation
# --------------------------------------------------------------------------------------
def router_fwd(logits, k, score_fn, *, expert_bias=None, valid_mask=None, scaling=1.0, want_stats=False,
               want_lse=False):
    """logits fp32 [T, E] -> dict(topk_idx int32 [T,k], topk_prob fp32 [T,k], counts int32 [E],
    aux_counts int32 [E], score_sum fp32 [E], lse fp32 [T])."""
    T, E = logits.shape
    assert logits.dtype == torch.float32 and logits.is_contiguous()
    dev = logits.device
    idx = torch.empty(T, k, dtype=torch.int32, device=dev)
    prob = torch.empty(T, k, dtype=torch.float32, device=dev)
    counts = torch.zeros(E, dtype=torch.int32, device=dev)
    grid = max(1, min((T + 7) // 8, 2 * num_sms(dev.index)))
    lse = torch.empty(T, dtype=torch.float32, device=dev) if (want_lse or want_stats) else None
    if want_stats:
        partial = torch.empty(grid, E, dtype=torch.float32, device=dev)
        score_sum = torch.empty(E, dtype=torch.float32, device=dev)
        aux_counts = torch.zeros(E, dtype=torch.int32, device=dev)
    else:
        partial = score_sum = aux_counts = None
    vm = valid_mask.to(torch.uint8).contiguous() if valid_mask is not None else None
    _check(lib().ttb_router_fwd(_p(logits), _p(expert_bias), _p(vm), _p(idx), _p(prob), _p(lse), _p(partial),
                                _p(score_sum), _p(aux_counts), _p(counts), C.c_longlong(T), C.c_int(E), C.c_int(k),
                                C.c_int(SCORE_FN[score_fn]), C.c_float(scaling), C.c_int(grid), _stream()),
           "ttb_router_fwd")
    return dict(topk_idx=idx, topk_prob=prob, counts=counts, aux_counts=aux_counts, score_sum=score_sum, lse=lse)


def router_bwd(logits, topk_idx, topk_prob, k, score_fn, *, dprob=None, aux_grad=None, lse=None, valid_mask=None,
               dlse=None, scaling=1.0):
    """d(logits) from the gradients of the routing weights (`dprob` [T,k]), of the per-expert score sums
    (`aux_grad` [E], applied to valid tokens) and of the per-token logsumexp (`dlse` [T])."""
    T, E = logits.shape
    dlogits = torch.empty_like(logits)
    vm = valid_mask.to(torch.uint8).contiguous() if valid_mask is not None else None
    _check(lib().ttb_router_bwd(_p(logits), _p(topk_idx), _p(topk_prob), _p(dprob), _p(aux_grad), _p(lse), _p(vm),
                                _p(dlse), _p(dlogits), C.c_longlong(T), C.c_int(E), C.c_int(k),
                                C.c_int(SCORE_FN[score_fn]), C.c_float(scaling), _stream()), "ttb_router_bwd")
    return dlogits


def aux_loss(score_sum: torch.Tensor, counts: torch.Tensor, k: int, scale_num: float, coeff: float):
    """Load-balance loss from the routing kernel's statistics.  Returns (out [2] = (aux, aux / coeff), d aux / d score_sum [E])."""
    E = score_sum.numel()
    out = torch.empty(2, dtype=torch.float32, device=score_sum.device)
    coef = torch.empty(E, dtype=torch.float32, device=score_sum.device)
    _check(lib().ttb_aux_loss(_p(score_sum), _p(counts), C.c_int(E), C.c_int(k), C.c_float(scale_num), C.c_float(coeff),
                              _p(out), _p(coef), _stream()), "ttb_aux_loss")
    return out, coef


def perm_index(topk_idx: torch.Tensor, num_experts: int, m_tiles_cap: int | None = None):
    """Padded (expert, token) permutation of the [T, k] expert ids.

    Returns dict(counts [E], seg_start [E+1], tile_group [m_tiles_cap], row_of [T*k], status [1], capacity_rows).
    All int32 device tensors; nothing is synchronised with the host.
    """
    idx = topk_idx.reshape(-1)
    assert idx.dtype == torch.int32 and idx.is_contiguous()
    N = idx.numel()
    dev = idx.device
    if m_tiles_cap is None:
        m_tiles_cap = (N + SEG_ALIGN - 1) // SEG_ALIGN + num_experts
    counts = torch.empty(num_experts, dtype=torch.int32, device=dev)
    seg_start = torch.empty(num_experts + 1, dtype=torch.int32, device=dev)
    tile_group = torch.empty(m_tiles_cap, dtype=torch.int32, device=dev)
    row_of = torch.empty(N, dtype=torch.int32, device=dev)
    st = torch.zeros(1, dtype=torch.int32, device=dev)
    _check(lib().ttb_perm_index(_p(idx), C.c_longlong(N), C.c_int(num_experts), _p(counts), _p(seg_start),
                                _p(tile_group), C.c_int(m_tiles_cap), _p(row_of), _p(st), _stream()),
           "ttb_perm_index")
    return dict(counts=counts, seg_start=seg_start, tile_group=tile_group, row_of=row_of, status=st,
                capacity_rows=m_tiles_cap * SEG_ALIGN)


def perm_scatter(src, row_of, k, capacity_rows, *, counts=None, seg_start=None, val=None, out=None):
    """dst[row_of[n]] = src[n // k]; pad rows of every expert segment are zeroed.  Returns (dst, row_val)."""
    T, H = src.shape
    N = row_of.numel()
    if out is None:
        out = torch.empty(capacity_rows, H, dtype=src.dtype, device=src.device)
    row_val = torch.empty(capacity_rows, dtype=torch.float32, device=src.device) if val is not None else None
    E = counts.numel() if counts is not None else 0
    _check(lib().ttb_perm_scatter(_p(src), C.c_longlong(src.stride(0)), _p(out), C.c_longlong(out.stride(0)),
                                  _p(row_of), _p(val), _p(row_val), C.c_void_p(0), _p(counts), _p(seg_start),
                                  C.c_int(E), C.c_longlong(N), C.c_int(k), C.c_int(H), _stream()), "ttb_perm_scatter")
    return out, row_val


def perm_combine(src, row_of, T, k, *, weights=None, residual=None):
    """out[t] = sum_j weights[t, j] * src[row_of[t*k+j]] (+ residual[t])."""
    H = src.shape[1]
    out = torch.empty(T, H, dtype=src.dtype, device=src.device)
    _check(lib().ttb_perm_combine(_p(src), C.c_longlong(src.stride(0)), _p(row_of), _p(weights), _p(residual),
                                  C.c_longlong(residual.stride(0) if residual is not None else 0), _p(out),
                                  C.c_longlong(out.stride(0)), C.c_longlong(T), C.c_int(k), C.c_int(H), _stream()),
           "ttb_perm_combine")
    return out


# --------------------------------------------------------------------------------------
# Flash attention (varlen, head_dim 128)
# --------------------------------------------------------------------------------------
def attn_status(reset: bool = False) -> tuple[int, int]:
    buf = (C.c_uint * 4)()
    _check(lib().ttb_attn_status(buf, C.c_int(1 if reset else 0)), "ttb_gemm_status")
    return int(buf[0]), int(buf[1])


def build_kv_tiles(cu_seqlens, block: int = 128) -> torch.Tensor:
    """Table of 128-row KV tiles for the backward pass, earliest tile of a document first (under a causal mask the
    earliest KV tiles are seen by the most query tiles, so they carry the most work)."""
    return torch.tensor(kv_tile_rows(cu_seqlens, block), dtype=torch.int32).reshape(-1, 3)


def kv_tile_rows(cu_seqlens, block: int = 128) -> list:
    offs = cu_seqlens.tolist() if isinstance(cu_seqlens, torch.Tensor) else list(cu_seqlens)
    rows = [(k0, a, b) for a, b in zip(offs[:-1], offs[1:]) for k0 in range(a, b, block)]
    rows.sort(key=lambda r: r[0] - r[2])
    return rows


def build_q_tiles(cu_seqlens, block: int = 128) -> torch.Tensor:
    """Host-side table of 128-row query tiles `[n, 3] = (first row, document start, document end)` from packed
    boundaries (a CPU tensor or list); no device synchronisation is involved."""
    return torch.tensor(q_tile_rows(cu_seqlens, block), dtype=torch.int32).reshape(-1, 3)


def q_tile_rows(cu_seqlens, block: int = 128) -> list:
    offs = cu_seqlens.tolist() if isinstance(cu_seqlens, torch.Tensor) else list(cu_seqlens)
    rows = []
    for a, b in zip(offs[:-1], offs[1:]):
        # longest-first inside a document does not matter; later tiles of causal documents do more work, so
        # emit them first to shorten the tail of the launch
        for q0 in range(a + ((b - a - 1) // block) * block, a - 1, -block) if b > a else ():
            rows.append((q0, a, b))
    rows.sort(key=lambda r: r[1] - r[0])             # across documents too: the tiles with the most KV blocks first
    return rows


def attn_tile_rows(lens, heads: int, causal: bool, sms: int, width: int = 128) -> int:
    """Query rows that a thread block of the forward kernel takes (the `block` of `build_q_tiles`): two tiles of 128 rows where
    that is faster, one where the longest blocks of the launch, or the last of their waves, would then be what everything waits for.

    Compared are the estimates of both launches in thousands of clocks, the larger of two bounds: the work of an SM, and, since of
    the j * sms + 1 longest blocks one SM takes j + 1, that many times the shortest of these.  A kv block and a thread block cost,
    with one query tile and with two, 2.05 + 8 and 3.2 + 8 for query / key heads up to 128 wide, 2.05 + 10 and 3.8 + 9 for 192 (half
    as much again for the scores, and one V stage when both tiles are there).  Fitted to 680 measured launches (widths 64, 72, 128
    and 192, one to 32 documents of 17 to 16384 tokens, 1 to 128 heads): of what the better of the two takes the choice loses 0.1 %
    on average.  One tile / two in us: 16001 tokens x 40 heads 3383 / 2795, 192 wide 3346 / 3397; 8192 x 8 148 / 128, 192 wide
    150 / 147; 16384 x 4, 192 wide 285 / 299; 2048 x 16 26 / 34; 5 documents of 784 x 8, full attention 26 / 31 (160 longer blocks
    are two waves on 148 SMs, as are 280 shorter ones); 8 of 300 x 8 14 / 10."""
    per_kv, per_block = ((2.05, 3.2), (8.0, 8.0)) if width <= 128 else ((2.05, 3.8), (10.0, 9.0))

    def launch(step: int) -> float:
        cost, start = per_kv[step - 1], per_block[step - 1]
        blocks, of = [], {}                                          # of one head; of a document with so many tiles
        for n in lens:
            tiles = (n + 127) // 128
            if tiles not in of:
                # entry i of a causal document sees min(step (i + 1), tiles) kv blocks, each entry of a full one all of them
                seen = range(step, tiles + step, step) if causal else [tiles] * ((tiles + step - 1) // step)
                of[tiles] = [min(kv, tiles) * cost + start for kv in seen]
            blocks += of[tiles]
        blocks.sort(reverse=True)
        waves = [(j + 1) * blocks[first // heads] for j, first in enumerate(range(0, len(blocks) * heads, sms))]
        return max(sum(blocks) * heads / sms, *waves, 0.0)

    return 256 if launch(2) < launch(1) else 128


def _covered(rows) -> tuple[int, int]:
    """(first, one past the last) covered row, or a negative first for unknown."""
    return rows if rows is not None else (-1, -1)


def attn_fwd(q, k, v, q_tiles_dev, *, scale: float, causal: bool = True, want_lse: bool = True,
             want_max_logit: bool = False, rows=None, tile_rows: int = 128):
    """q: [T, Hq, D]; k: [T, Hk, D]; v: [T, Hk, Dv] (may be a row-strided view), D and Dv up to 128 in multiples of 8, or D = 192
    with Dv = 128 (multi-head latent attention).  `q_tiles_dev`: `build_q_tiles(cu, tile_rows)`, one thread block per entry and query head, with
    `tile_rows` 128 or 256.  `rows` (optional): (first, one past the last) row that the tile table covers; the kernel writes
    every one of them.  Returns (out [T, Hq, Dv], lse [Hq, T], max_logit [Hq])."""
    return host().attn_fwd(q, k, v, q_tiles_dev, scale, causal, want_lse, want_max_logit, *_covered(rows), tile_rows)


def delta_state_scan(a_tiles, b_tiles, u, decay, init, add, seq_chunks_dev, *, reverse: bool, s1: float, s2: float, zero_first: bool = False,
                     longest: int = 0):
    """Chunk-state recurrence of the delta rule (csrc/delta_state.cu).  `a_tiles`, `b_tiles`: bf16 [H, NC, 64, 128];
    `u`: fp32 [H, NC, 64, 128]; `decay`: fp32 [H, NC] or [H, NC, 128]; `init`: fp32 [H, nseq, 128, 128] or None;
    `add`: fp32 [H, NC + nseq, 128, 128] (required when `reverse`); `seq_chunks_dev`: int32 [nseq, 2].  A reverse pass starts from the
    last slots of `add`, with `zero_first` from zero (those slots are not read).
    ``longest``: chunks of the longest sequence, which the choice between the kernel's forms goes by (0: not known).
    Returns (x fp32 [H, NC, 64, 128], states fp32 [H, NC + nseq, 128, 128])."""
    return host().delta_state_scan(a_tiles, b_tiles, u, decay, init, add, seq_chunks_dev, (2 if zero_first else 1) if reverse else 0, s1, s2,
                                   longest)


# Inputs of the chunk kernels: v: bf16 [rows, H, 128]; q, k: the same or, with one decay per head, of H / rep heads that serve rep value
# heads each (any row / head stride that keeps 16-byte alignment); g: fp32 [rows, H] or [rows, H, 128] (one decay per head, or per head
# and channel); beta: fp32 [rows, H]; chunk_rows: int32 [NC, 3] on the device (first row, number of rows, sequence of every chunk).
def delta_prep(q, k, v, g, beta, chunk_rows, *, l2: bool, scale: float):
    """Chunk-parallel operands of the gated delta rule (csrc/delta_chunk.cu).  Returns (T, A fp32 [H, NC, 64, 64],
    u fp32 [H, NC, 64, 128], w, k_out bf16 [H, NC, 64, 128], decay fp32 [H, NC] or [H, NC, 128])."""
    return host().delta_prep(q, k, v, g, beta, chunk_rows, l2, scale)


def delta_out(q, k, v, g, beta, chunk_rows, A, x, states, *, l2: bool, scale: float):
    """o bf16 [rows, H, 128] from the new values `x` and the chunk-start states of the recurrence."""
    return host().delta_out(q, k, v, g, beta, chunk_rows, A, x, states, l2, scale)


def delta_bwd_pre(q, k, v, g, beta, chunk_rows, do, A, nseq: int, *, l2: bool, scale: float):
    """Gradients that reach the recurrence directly: (gx like x, gS [H, NC + nseq, 128, 128]; the slots behind the last
    chunk of a sequence are left to the caller)."""
    return host().delta_bwd_pre(q, k, v, g, beta, chunk_rows, do, A, nseq, l2, scale)


class _DeltaChunkIn(C.Structure):
    """`struct DeltaChunkIn` of csrc/entries.h."""

    _fields_ = [("q", C.c_void_p), ("k", C.c_void_p), ("v", C.c_void_p),
                ("q_t", C.c_longlong), ("q_h", C.c_longlong), ("k_t", C.c_longlong), ("k_h", C.c_longlong),
                ("v_t", C.c_longlong), ("v_h", C.c_longlong),
                ("g", C.c_void_p), ("beta", C.c_void_p), ("chunk_rows", C.c_void_p),
                ("H", C.c_int), ("NC", C.c_int), ("l2", C.c_int), ("scale", C.c_float), ("rep", C.c_int)]


def delta_bwd_post(q, k, v, g, beta, chunk_rows, do, T, x, dx, states, dstates, *, l2: bool, scale: float):
    """(dq, dk bf16 like q, dv bf16 [rows, H, 128], dg like g, dbeta fp32 [rows, H])."""
    R, H, _ = v.shape
    Hk, NC = q.shape[1], chunk_rows.shape[0]
    check_device(q)
    for t, heads in ((q, Hk), (k, Hk), (v, H)):
        assert t.dtype == torch.bfloat16 and t.shape == (R, heads, 128) and t.stride(2) == 1
    assert H % Hk == 0 and (Hk == H or g.dim() == 2)
    assert g.dtype == torch.float32 and g.shape in ((R, H), (R, H, 128)) and g.is_contiguous()
    assert beta.dtype == torch.float32 and beta.shape == (R, H) and beta.is_contiguous()
    assert chunk_rows.dtype == torch.int32 and chunk_rows.is_contiguous() and chunk_rows.shape[1] == 3
    a = _DeltaChunkIn(q.data_ptr(), k.data_ptr(), v.data_ptr(), q.stride(0), q.stride(1), k.stride(0), k.stride(1), v.stride(0), v.stride(1),
                      g.data_ptr(), beta.data_ptr(), chunk_rows.data_ptr(), H, NC, int(l2), scale, H // Hk)
    dq, dk, dv = (torch.empty(v.shape, dtype=torch.bfloat16, device=q.device) for _ in range(3))   # of every value head
    dg, dbeta = torch.empty_like(g), torch.empty_like(beta)
    # held until the launches are queued: a pointer alone would let another thread of this stream be given the block first
    scratch = torch.empty(4, *x.shape, dtype=torch.float32, device=q.device) if g.dim() == 3 else None
    name = "ttb_delta_vec_bwd_post" if g.dim() == 3 else "ttb_delta_bwd_post"
    _check(getattr(lib(), name)(C.byref(a), _p(do), _p(T), _p(x), _p(dx), _p(states), _p(dstates), C.c_int(states.shape[1] - NC),
                                _p(dq), _p(dk), _p(dv), _p(dg), _p(dbeta), *([_p(scratch)] if scratch is not None else []), _stream()), name)
    if H > Hk:
        per_head, (dq, dk) = (dq, dk), (torch.empty(q.shape, dtype=torch.bfloat16, device=q.device) for _ in range(2))
        _check(lib().ttb_delta_head_sum(_p(per_head[0]), _p(per_head[1]), _p(dq), _p(dk), C.c_longlong(R * Hk), C.c_int(H // Hk), _stream()),
               "ttb_delta_head_sum")
    return dq, dk, dv, dg, dbeta


# --------------------------------------------------------------------------------------
# Expert-parallel exchange over peer memory (see csrc/comm.cu)
# --------------------------------------------------------------------------------------
def comm_status(reset: bool = False) -> tuple[int, int]:
    buf = (C.c_uint * 4)()
    _check(lib().ttb_comm_status(buf, C.c_int(1 if reset else 0)), "ttb_gemm_status")
    return int(buf[0]), int(buf[1])


def perm_rank(idx: torch.Tensor, num_experts: int, base: torch.Tensor) -> torch.Tensor:
    flat = idx.reshape(-1)
    row_of = torch.empty_like(flat)
    _check(lib().ttb_perm_rank(_p(flat), C.c_longlong(flat.numel()), C.c_int(num_experts), _p(base), _p(row_of), _stream()),
           "ttb_perm_rank")
    return row_of


def perm_zero_pad(dst, counts, seg_start, row_val=None):
    _check(lib().ttb_perm_zero_pad(_p(dst), C.c_longlong(dst.stride(0)), _p(counts), _p(seg_start), _p(row_val),
                                   C.c_int(counts.numel()), C.c_int(dst.shape[1]), _stream()), "ttb_perm_zero_pad")


def ep_exchange(peer_ptrs, off_counts, off_flags, counts, rank, world, num_experts, epoch, budget_ms, m_tiles_cap,
                status):
    dev = counts.device
    El = num_experts // world
    seg_start = torch.empty(El + 1, dtype=torch.int32, device=dev)
    recv_counts = torch.empty(El, dtype=torch.int32, device=dev)
    tile_group = torch.empty(m_tiles_cap, dtype=torch.int32, device=dev)
    dest_base = torch.empty(num_experts, dtype=torch.int32, device=dev)
    _check(lib().ttb_ep_exchange(peer_ptrs, C.c_longlong(off_counts), C.c_longlong(off_flags), _p(counts), C.c_int(rank),
                                 C.c_int(world), C.c_int(num_experts), C.c_int(epoch), C.c_longlong(budget_ms),
                                 C.c_int(m_tiles_cap), _p(seg_start), _p(recv_counts), _p(tile_group), _p(dest_base),
                                 _p(status), _stream()), "ttb_ep_exchange")
    return seg_start, recv_counts, tile_group, dest_base


class _EpDispatchArgs(C.Structure):
    _fields_ = [
        ("peer_ptrs", C.c_void_p),
        ("off_counts", C.c_longlong), ("off_flags_counts", C.c_longlong), ("off_rows", C.c_longlong),
        ("off_vals", C.c_longlong), ("off_flags_rows", C.c_longlong),
        ("counts", C.c_void_p), ("expert", C.c_void_p), ("src", C.c_void_p), ("lds", C.c_longlong), ("val", C.c_void_p),
        ("recv_rows_local", C.c_void_p), ("recv_vals_local", C.c_void_p),
        ("seg_start", C.c_void_p), ("recv_counts", C.c_void_p), ("tile_group", C.c_void_p), ("dest_base", C.c_void_p),
        ("dest_row", C.c_void_p), ("done_counter", C.c_void_p), ("status", C.c_void_p),
        ("N", C.c_longlong), ("cap_rows", C.c_longlong), ("budget_ms", C.c_longlong),
        ("rank", C.c_int), ("W", C.c_int), ("E", C.c_int), ("k", C.c_int), ("H", C.c_int), ("m_tiles_cap", C.c_int),
        ("epoch_counts", C.c_int), ("epoch_rows", C.c_int), ("grid", C.c_int), ("exchange", C.c_int),
    ]


def ep_dispatch_all(peer_ptrs, *, off_counts, off_flags_counts, off_rows, off_vals, off_flags_rows, counts, expert, src, val,
                    recv_rows_local, recv_vals_local, rank, world, num_experts, k, m_tiles_cap, cap_rows, epoch_counts,
                    epoch_rows, budget_ms, done_counter, status, tables=None):
    """Expert-parallel row dispatch in one host call.  With `tables=None`: counts exchange, destination rows, padding
    zeroed, scatter, landed wait; returns (seg_start, recv_counts, tile_group, dest_row).  With `tables = (seg_start,
    recv_counts, dest_row)` (backward of combine) only the last three stages run."""
    dev = src.device
    N = expert.numel()
    El = num_experts // world
    a = _EpDispatchArgs()
    if tables is None:
        seg_start = torch.empty(El + 1, dtype=torch.int32, device=dev)
        recv_counts = torch.empty(El, dtype=torch.int32, device=dev)
        tile_group = torch.empty(m_tiles_cap, dtype=torch.int32, device=dev)
        dest_base = torch.empty(num_experts, dtype=torch.int32, device=dev)
        dest_row = torch.empty_like(expert)
        a.exchange, a.counts = 1, counts.data_ptr()
        a.tile_group, a.dest_base = tile_group.data_ptr(), dest_base.data_ptr()
    else:
        seg_start, recv_counts, dest_row = tables
        tile_group = None
        a.exchange = 0
    a.peer_ptrs = C.addressof(peer_ptrs)
    a.off_counts, a.off_flags_counts, a.off_rows = off_counts, off_flags_counts, off_rows
    a.off_vals, a.off_flags_rows = off_vals, off_flags_rows
    a.expert, a.src, a.lds = expert.data_ptr(), src.data_ptr(), src.stride(0)
    a.val = val.data_ptr() if val is not None else None
    a.recv_rows_local = recv_rows_local.data_ptr()
    a.recv_vals_local = recv_vals_local.data_ptr() if recv_vals_local is not None else None
    a.seg_start, a.recv_counts, a.dest_row = seg_start.data_ptr(), recv_counts.data_ptr(), dest_row.data_ptr()
    a.done_counter, a.status = done_counter.data_ptr(), status.data_ptr()
    a.N, a.cap_rows, a.budget_ms = N, cap_rows, budget_ms
    a.rank, a.W, a.E, a.k, a.H, a.m_tiles_cap = rank, world, num_experts, k, src.shape[1], m_tiles_cap
    a.epoch_counts, a.epoch_rows = epoch_counts, epoch_rows
    a.grid = max(1, min((N + 7) // 8, 8 * num_sms(dev.index)))
    _check(lib().ttb_ep_dispatch_all(C.byref(a), _stream()), "ttb_ep_dispatch_all" if tables is None else "ttb_ep_dispatch_rows")
    return seg_start, recv_counts, tile_group, dest_row


def ep_combine_all(peer_ptrs, *, off_rows, off_vals, off_flags, expert, dest_row, T, k, H, El, rank, world, epoch, budget_ms,
                   cap_rows, status, residual=None, want_vals=False):
    """Ready signal, ready wait and the k-way gather (optionally also the per-entry scalars) in one host call."""
    dev = expert.device
    out = torch.empty(T, H, dtype=torch.bfloat16, device=dev)
    vals = torch.empty(T * k, dtype=torch.float32, device=dev) if want_vals else None
    _check(lib().ttb_ep_combine_all(peer_ptrs, C.c_longlong(off_rows), C.c_longlong(off_vals), C.c_longlong(off_flags),
                                    _p(expert), _p(dest_row), _p(residual),
                                    C.c_longlong(residual.stride(0) if residual is not None else 0), _p(out),
                                    C.c_longlong(out.stride(0)), _p(vals), C.c_longlong(T), C.c_int(k), C.c_int(H),
                                    C.c_int(El), C.c_int(rank), C.c_int(world), C.c_int(epoch), C.c_longlong(budget_ms),
                                    C.c_longlong(cap_rows), _p(status), _stream()),
           "ttb_ep_combine_vals" if want_vals else "ttb_ep_combine_all")
    return out, vals


class _EpPrepareArgs(C.Structure):
    _fields_ = [
        ("peer_ptrs", C.c_void_p), ("off_counts", C.c_longlong), ("off_flags_counts", C.c_longlong),
        ("counts", C.c_void_p), ("expert", C.c_void_p),
        ("recv_rows_local", C.c_void_p), ("recv_vals_local", C.c_void_p), ("recv_tags_local", C.c_void_p),
        ("seg_start", C.c_void_p), ("recv_counts", C.c_void_p), ("tile_group", C.c_void_p), ("dest_base", C.c_void_p),
        ("dest_row", C.c_void_p), ("send_base", C.c_void_p), ("order", C.c_void_p),
        ("sent", C.c_void_p), ("status", C.c_void_p),
        ("N", C.c_longlong), ("budget_ms", C.c_longlong),
        ("rank", C.c_int), ("W", C.c_int), ("E", C.c_int), ("H", C.c_int), ("m_tiles_cap", C.c_int),
        ("epoch_counts", C.c_int), ("exchange", C.c_int),
    ]


def ep_prepare(peer_ptrs, *, off_counts, off_flags_counts, counts, expert, recv_rows, recv_vals, recv_tags, sent, status,
               rank, world, num_experts, m_tiles_cap, epoch_counts, budget_ms, tables=None):
    """Everything a fused expert-parallel GEMM needs before it starts, in one host call.  Forward (`tables=None`):
    counts exchange with the peers, layout tables, destination row and send order of every entry, padding rows of the
    receive buffer cleared; returns `(seg_start, recv_counts, tile_group, dest_row, order)`.  Backward (`tables =
    (seg_start, recv_counts)` of the forward pass): only the receive buffer is prepared again."""
    dev = expert.device
    N = expert.numel()
    El = num_experts // world
    a = _EpPrepareArgs()
    if tables is None:
        # one int32 block: seg_start [El+1] | recv_counts [El] | tile_group [cap] | dest_base [E] | send_base [E]
        meta = torch.empty(2 * El + 1 + m_tiles_cap + 2 * num_experts, dtype=torch.int32, device=dev)
        seg_start, recv_counts = meta[:El + 1], meta[El + 1:2 * El + 1]
        o = 2 * El + 1
        tile_group = meta[o:o + m_tiles_cap]
        dest_base, send_base = meta[o + m_tiles_cap:o + m_tiles_cap + num_experts], meta[o + m_tiles_cap + num_experts:]
        rows = torch.empty(2, N, dtype=torch.int32, device=dev)
        dest_row, order = rows[0], rows[1]
        a.exchange, a.counts = 1, counts.data_ptr()
        a.tile_group, a.dest_base, a.send_base = tile_group.data_ptr(), dest_base.data_ptr(), send_base.data_ptr()
        a.dest_row, a.order = dest_row.data_ptr(), order.data_ptr()
    else:
        seg_start, recv_counts = tables
        tile_group = dest_row = order = None
        a.exchange = 0
    a.peer_ptrs = C.addressof(peer_ptrs)
    a.off_counts, a.off_flags_counts = off_counts, off_flags_counts
    a.expert = expert.data_ptr()
    a.recv_rows_local, a.recv_vals_local, a.recv_tags_local = recv_rows.data_ptr(), recv_vals.data_ptr(), recv_tags.data_ptr()
    a.seg_start, a.recv_counts = seg_start.data_ptr(), recv_counts.data_ptr()
    a.sent, a.status = sent.data_ptr(), status.data_ptr()
    a.N, a.budget_ms = N, budget_ms
    a.rank, a.W, a.E, a.H, a.m_tiles_cap = rank, world, num_experts, recv_rows.shape[1], m_tiles_cap
    a.epoch_counts = epoch_counts
    _check(lib().ttb_ep_prepare(C.byref(a), _stream()), "ttb_ep_prepare" if tables is None else "ttb_ep_prepare_bwd")
    return seg_start, recv_counts, tile_group, dest_row, order


def ep_save(recv_rows, recv_vals, seg_start, El):
    """Copies the rows (and their scalars) that landed in the receive buffer; the row count is read on the device."""
    cap, H = recv_rows.shape
    rows = torch.empty_like(recv_rows)
    vals = torch.empty_like(recv_vals) if recv_vals is not None else None
    grid = 4 * num_sms(recv_rows.device.index)
    _check(lib().ttb_ep_save(_p(recv_rows), _p(rows), _p(recv_vals), _p(vals), _p(seg_start), C.c_int(El), C.c_int(H),
                             C.c_longlong(cap), C.c_int(grid), _stream()), "ttb_ep_save")
    return rows, vals


def ep_ksum(peer_ptrs, off_ret, off_ret_flags, T, k, H, world, rank, epoch, budget_ms, status, residual=None):
    """Waits for every owner's "rows returned" flag, then sums the k returned rows of every token (+ residual)."""
    out = torch.empty(T, H, dtype=torch.bfloat16, device=status.device)
    _check(lib().ttb_ep_ksum(peer_ptrs, C.c_longlong(off_ret), C.c_longlong(off_ret_flags), _p(residual),
                             C.c_longlong(residual.stride(0) if residual is not None else 0), _p(out),
                             C.c_longlong(out.stride(0)), C.c_longlong(T), C.c_int(k), C.c_int(H), C.c_int(world),
                             C.c_int(rank), C.c_int(epoch), C.c_longlong(budget_ms), _p(status), _stream()), "ttb_ep_ksum")
    return out


def ep_scatter(peer_ptrs, off_rows, off_vals, off_flags, src, expert, dest_row, val, k, El, rank, world, epoch, cap_rows,
               done_counter, status):
    N = expert.numel()
    grid = max(1, min((N + 7) // 8, 8 * num_sms(src.device.index)))
    _check(lib().ttb_ep_scatter(peer_ptrs, C.c_longlong(off_rows), C.c_longlong(off_vals), C.c_longlong(off_flags), _p(src),
                                C.c_longlong(src.stride(0)), _p(expert), _p(dest_row), _p(val), C.c_longlong(N), C.c_int(k),
                                C.c_int(src.shape[1]), C.c_int(El), C.c_int(rank), C.c_int(world), C.c_int(epoch),
                                C.c_longlong(cap_rows), _p(done_counter), _p(status), C.c_int(grid), _stream()),
           "ttb_ep_scatter")


def flag_signal(peer_ptrs, off_flags, rank, world, epoch):
    _check(lib().ttb_flag_signal(peer_ptrs, C.c_longlong(off_flags), C.c_int(rank), C.c_int(world), C.c_int(epoch),
                                 _stream()), "ttb_flag_signal")


def flag_wait(peer_ptrs, off_flags, rank, world, epoch, budget_ms, status):
    _check(lib().ttb_flag_wait(peer_ptrs, C.c_longlong(off_flags), C.c_int(rank), C.c_int(world), C.c_int(epoch),
                               C.c_longlong(budget_ms), _p(status), _stream()), "ttb_flag_wait")


def ep_gather(peer_ptrs, off_rows, expert, dest_row, T, k, H, El, world, cap_rows, status, *, weights=None, residual=None,
              dtype=torch.bfloat16):
    out = torch.empty(T, H, dtype=dtype, device=expert.device)
    _check(lib().ttb_ep_gather(peer_ptrs, C.c_longlong(off_rows), _p(expert), _p(dest_row), _p(weights), _p(residual),
                               C.c_longlong(residual.stride(0) if residual is not None else 0), _p(out),
                               C.c_longlong(out.stride(0)), C.c_longlong(T), C.c_int(k), C.c_int(H), C.c_int(El),
                               C.c_int(world), C.c_longlong(cap_rows), _p(status), _stream()), "ttb_ep_gather")
    return out


def ep_gather_vals(peer_ptrs, off_vals, expert, dest_row, El, world, cap_rows, status):
    N = expert.numel()
    out = torch.empty(N, dtype=torch.float32, device=expert.device)
    _check(lib().ttb_ep_gather_vals(peer_ptrs, C.c_longlong(off_vals), _p(expert), _p(dest_row), _p(out), C.c_longlong(N),
                                    C.c_int(El), C.c_int(world), C.c_longlong(cap_rows), _p(status), _stream()),
           "ttb_ep_gather_vals")
    return out


def attn_bwd(dout, q, k, v, out, lse, kv_tiles_dev, *, scale: float, causal: bool = True, q_tiles_dev=None,
             deterministic: bool = False, rows=None):
    """Gradients of `attn_fwd`.  Returns (dq [T,Hq,D], dk [T,Hk,D], dv [T,Hk,Dv]) in bf16; `rows` as in `attn_fwd`.

    Heads up to 128 wide by default: one kernel; dQ tiles are added into an fp32 scratch buffer by TMA reductions and, with
    grouped-query attention, the dK / dV of a group's query heads are summed with atomics (the order of the adds is not
    fixed).  For 192-wide query / key heads that kernel computes dK / dV only and dQ comes from the query-major pass
    (`q_tiles_dev` required), which writes every dQ tile once.  `deterministic=True` uses that split for every width
    and lets one CTA per kv head walk the query heads of its group, so nothing is reduced with atomics and the result
    is bit-reproducible."""
    return host().attn_bwd(dout, q, k, v, out, lse, kv_tiles_dev, scale, causal, q_tiles_dev, deterministic, *_covered(rows))


# --------------------------------------------------------------------------------------
# Ulysses sequence parallelism over peer memory
# --------------------------------------------------------------------------------------
def ulysses_qkv_scatter(peer_ptrs, off_q, off_k, off_v, off_flags, qkv, n_q, n_kv, rep, wq, wk, cos, sin, eps, rank, world,
                        epoch, done_counter, use_norm=True):
    """Per-head RMSNorm + RoPE of the q / k columns of `qkv` [Tl, (n_q + 2 n_kv) * 128] and a copy of the v columns,
    stored straight into the owning ranks' `[T, heads / world, 128]` buffers; publishes this rank's "landed" flag.
    Returns rstd [Tl * (n_q + n_kv)]."""
    Tl = qkv.shape[0]
    check_device(qkv)
    rstd = torch.empty(Tl * (n_q + n_kv), dtype=torch.float32, device=qkv.device)
    warps = Tl * (n_q + 2 * n_kv)
    grid = max(1, min((warps + 7) // 8, 8 * num_sms(qkv.device.index)))
    _check(lib().ttb_ulysses_qkv_scatter(peer_ptrs, C.c_longlong(off_q), C.c_longlong(off_k), C.c_longlong(off_v),
                                         C.c_longlong(off_flags), _p(qkv), C.c_longlong(qkv.stride(0)), _p(wq), _p(wk),
                                         _p(cos), _p(sin), _p(rstd), C.c_longlong(Tl), C.c_int(n_q), C.c_int(n_kv),
                                         C.c_int(rep), C.c_int(world), C.c_int(rank), C.c_int(epoch),
                                         C.c_int(int(use_norm)), C.c_float(eps), _p(done_counter), C.c_int(grid),
                                         _stream()), "ttb_ulysses_qkv_scatter")
    return rstd


def ulysses_move(peer_ptrs, off_buf, off_flags, local, heads, rep, rank, world, epoch, done_counter, status, gather: bool):
    """`gather=False`: push `local` [Tl, heads, 128] into the owners' buffers and publish the "landed" flag.
    `gather=True`: fill `local` from the owners' buffers (replicas summed)."""
    Tl = local.shape[0]
    check_device(local)
    assert local.is_contiguous() and local.dtype == torch.bfloat16 and local.shape[-1] == 128
    grid = max(1, min((Tl * heads + 7) // 8, 8 * num_sms(local.device.index)))
    _check(lib().ttb_ulysses_move(peer_ptrs, C.c_longlong(off_buf), C.c_longlong(off_flags), _p(local), C.c_longlong(Tl),
                                  C.c_int(heads), C.c_int(rep), C.c_int(world), C.c_int(rank), C.c_int(epoch),
                                  _p(done_counter), _p(status), C.c_int(int(gather)), C.c_int(grid), _stream()),
           "ttb_ulysses_move")
    return local


def multimem_allreduce_f32(mc_ptr: int, n: int, rank: int, world: int, scale: float = 1.0, grid: int = 296):
    """In-switch all-reduce (sum, then `scale`) of `n` fp32 values at multicast address `mc_ptr`; this rank handles slice
    `rank`.  The caller synchronises the ranks before (all inputs written) and after (all slices stored)."""
    _check(lib().ttb_multimem_allreduce_f32(C.c_void_p(mc_ptr), C.c_longlong(n), C.c_int(rank), C.c_int(world), C.c_float(scale),
                                            C.c_int(grid), _stream()), "ttb_multimem_allreduce_f32")


def peer_collective(peer_ptrs, off_data, off_ready, off_consumed, units, rank, world, epoch, budget_ms, done_counter,
                    status, *, kind: int, out: torch.Tensor | None = None, scale: float = 1.0, grid: int = 64):
    """Pull all-gather (kind 0) or pull reduce-scatter of fp32 (kind 1) / bf16 (kind 2) pieces over a slot of the
    symmetric buffer; `units` is the piece length in 16-byte units."""
    _check(lib().ttb_peer_collective(peer_ptrs, C.c_longlong(off_data), C.c_longlong(off_ready),
                                     C.c_longlong(off_consumed), C.c_longlong(units), C.c_int(rank), C.c_int(world),
                                     C.c_int(epoch), C.c_longlong(budget_ms), C.c_float(scale), _p(out),
                                     _p(done_counter), _p(status), C.c_int(kind), C.c_int(grid), _stream()),
           "ttb_peer_collective")
