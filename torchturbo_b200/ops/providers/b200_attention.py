"""tcgen05 variable-length flash attention as the `attention` / `attention_with_max_logits` operators."""
from __future__ import annotations

import math
import os

import torch

from ... import kernels as K
from ...runtime import TurboDevice
from ...utils.functools import cache
from ..base import OpImplKind
from ..registry import register_op
from . import native as N
from .b200 import BF16, _aligned, _B200Op, _ok


class _Tiles:
    """Tile tables of one batch on the device: query tiles of 128 rows and pairs of them, key tiles and the boundaries, in one
    copy from pinned memory (asynchronous), with what the host knows of the boundaries."""

    def __init__(self, cu_seqlens, device):
        offs = cu_seqlens.tolist()
        tables = K.q_tile_rows(offs), K.q_tile_rows(offs, 256), K.kv_tile_rows(offs)
        flat = torch.tensor([x for table in tables for row in table for x in row] + offs, dtype=torch.int32)
        *views, self.cu = flat.pin_memory().to(device, non_blocking=True).split([3 * len(t) for t in tables] + [len(offs)])
        q1, q2, self.kv = (v.view(-1, 3) for v in views)
        self.q = {128: q1, 256: q2}
        self.n_valid = offs[-1]
        # the tables cover [first, last) without holes when the boundaries do not decrease
        self.rows = (offs[0], offs[-1]) if all(a <= b for a, b in zip(offs[:-1], offs[1:])) else None
        self.lens = [max(b - a, 0) for a, b in zip(offs[:-1], offs[1:])]
        self._tile_rows: dict = {}

    def tile_rows(self, heads: int, causal: bool, width: int) -> int:
        key = (heads, causal, width > 128)
        if key not in self._tile_rows:
            self._tile_rows[key] = K.attn_tile_rows(self.lens, heads, causal, K.num_sms(self.cu.device.index), width)
        return self._tile_rows[key]


@cache
def _tiles_for(cu_seqlens, device) -> _Tiles:
    """Built once for a batch and shared by every layer."""
    return _Tiles(cu_seqlens, device)


class FlashAttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, cu_seqlens, max_seqlen, causal, scale, want_ml):
        tiles = _tiles_for(cu_seqlens, q.device)
        block = tiles.tile_rows(q.shape[1], causal, q.shape[2])
        out, lse, ml = K.attn_fwd(q, k, v, tiles.q[block], scale=scale, causal=causal, want_max_logit=want_ml, rows=tiles.rows,
                                  tile_rows=block)
        ctx.save_for_backward(q, k, v, out, lse)
        ctx.meta = (cu_seqlens, max_seqlen, causal, scale, tiles.n_valid)
        if want_ml:
            ctx.mark_non_differentiable(ml)
            return out, ml
        return out

    @staticmethod
    def backward(ctx, dout, *_):
        q, k, v, out, lse = ctx.saved_tensors
        cu_seqlens, max_seqlen, causal, scale, n = ctx.meta
        if not _library_backward():
            tiles = _tiles_for(cu_seqlens, q.device)
            dq, dk, dv = K.attn_bwd(_aligned(dout), q, k, v, out, lse, tiles.kv, scale=scale, causal=causal,
                                    q_tiles_dev=tiles.q[128], deterministic=torch.are_deterministic_algorithms_enabled(),
                                    rows=tiles.rows)
            return dq, dk, dv, None, None, None, None, None
        # library backward on this kernel's out / lse (selected with TORCHTURBO_ATTN_BWD=flash_attn2; used as a baseline)
        from flash_attn.flash_attn_interface import _flash_attn_varlen_backward

        cu = _tiles_for(cu_seqlens, q.device).cu
        if max_seqlen is None:
            max_seqlen = int((cu_seqlens[1:] - cu_seqlens[:-1]).max())
        dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros(k.shape, dtype=k.dtype, device=k.device)
        _flash_attn_varlen_backward(dout.contiguous()[:n], q[:n], k[:n], v[:n].contiguous(), out[:n], lse[:, :n].contiguous(),
                                    dq[:n], dk[:n], dv[:n], cu, cu, max_seqlen, max_seqlen, 0.0, scale, causal,
                                    -1, -1, 0.0, None, False)
        return dq, dk, dv, None, None, None, None, None


def _LIB_FALLBACK(q, k, v, cu_seqlens, max_seqlen, *, causal, scale):
    from .b200 import FlashAttn2Varlen

    lib = FlashAttn2Varlen()
    if lib.available():
        return lib(q, k, v, cu_seqlens, max_seqlen, causal=causal, scale=scale)
    return N.attention_ref(q, k, v, cu_seqlens, causal, scale)


def _library_backward() -> bool:
    return os.environ.get("TORCHTURBO_ATTN_BWD", "tcgen05") != "tcgen05"


def _narrow(q, k, v):
    """Head widths below 128 in multiples of 8 (ViT: 72, 80), which the kernels take as they are: the loads fill the tiles' missing
    columns with zeros."""
    widths = q.shape[-1], v.shape[-1]
    return _paddable(q, k, v) and min(widths) > 0 and not any(w % 8 for w in widths) and not _library_backward()


def _rows_of_heads(t):
    """[T, H, D] whose heads lie in a row and whose rows start on 16 bytes and do not overlap; copied only where they do not.  Goes
    by the strides: a tensor with one token or one head counts as contiguous whatever the stride of that dimension."""
    H, D = t.shape[1:]
    if t.stride(2) != 1 or t.stride(1) != D or t.stride(0) < H * D or t.stride(0) % 8 or t.data_ptr() % 16:
        t = t.clone(memory_format=torch.contiguous_format)
    return t


def _usable(q, k, v):
    """128-wide heads, or multi-head latent attention (query / key 192 wide, value 128 wide)."""
    return _ok(q, k, v) and q.shape[-1] in (128, 192) and k.shape[-1] == q.shape[-1] and v.shape[-1] == 128 and q.dim() == 3 \
        and q.shape[1] % k.shape[1] == 0 and v.stride(2) == 1 and v.stride(1) == 128


def _paddable(q, k, v):
    """Any head width below 128 can run on the 128-wide kernel with zero columns: padded query / key columns add
    nothing to the logits and padded value columns only produce output columns that are sliced away."""
    return _ok(q, k, v) and q.dim() == 3 and q.shape[1] % k.shape[1] == 0 and q.shape[-1] == k.shape[-1] and \
        q.shape[-1] <= 128 and v.shape[-1] <= 128 and (q.shape[-1] < 128 or v.shape[-1] < 128)


def _narrow_call(q, k, v, cu, max_seqlen, causal, scale, want_ml):
    import torch.nn.functional as F

    dqk, dv = q.shape[-1], v.shape[-1]
    scale = scale if scale is not None else 1.0 / math.sqrt(dqk)
    if _narrow(q, k, v):
        return FlashAttnFn.apply(_rows_of_heads(_aligned(q)), _rows_of_heads(_aligned(k)), _rows_of_heads(v),
                                 cu.cpu() if cu.is_cuda else cu, max_seqlen, causal, float(scale), want_ml)
    qp, kp, vp = F.pad(q, (0, 128 - dqk)), F.pad(k, (0, 128 - dqk)), F.pad(v, (0, 128 - dv))
    res = FlashAttnFn.apply(qp, kp, vp, cu.cpu() if cu.is_cuda else cu, max_seqlen, causal, float(scale), want_ml)
    if want_ml:
        return res[0][..., :dv], res[1]
    return res[..., :dv]


@register_op(op_name="attention", impl_name="tcgen05_varlen_attention", kind=OpImplKind.CUSTOM, priority=100,
             devices=(TurboDevice.CUDA,))
class B200Attention(_B200Op):
    def __call__(self, q, k, v, cu_seqlens, max_seqlen=None, *, causal=True, scale=None):
        cu = cu_seqlens if isinstance(cu_seqlens, torch.Tensor) else torch.tensor(cu_seqlens, dtype=torch.int32)
        if not _usable(q, k, v):
            if _paddable(q, k, v):
                return _narrow_call(q, k, v, cu, max_seqlen, causal, scale, False)
            # other head widths: the library kernel
            return _LIB_FALLBACK(q, k, v, cu_seqlens, max_seqlen, causal=causal, scale=scale)
        scale = scale if scale is not None else 1.0 / math.sqrt(q.shape[-1])
        return FlashAttnFn.apply(q.contiguous(), k.contiguous(), v, cu.cpu() if cu.is_cuda else cu, max_seqlen, causal,
                                 float(scale), False)


@register_op(op_name="attention_with_max_logits", impl_name="tcgen05_varlen_attention_max_logits",
             kind=OpImplKind.CUSTOM, priority=100, devices=(TurboDevice.CUDA,))
class B200AttentionWithMaxLogits(_B200Op):
    def __call__(self, q, k, v, cu_seqlens, max_seqlen=None, *, causal=True, scale=None):
        cu = cu_seqlens if isinstance(cu_seqlens, torch.Tensor) else torch.tensor(cu_seqlens, dtype=torch.int32)
        if not _usable(q, k, v):
            if _paddable(q, k, v):
                return _narrow_call(q, k, v, cu, max_seqlen, causal, scale, True)
            return N.attention_ref(q, k, v, cu_seqlens, causal, scale, want_max_logits=True)
        scale = scale if scale is not None else 1.0 / math.sqrt(q.shape[-1])
        return FlashAttnFn.apply(q.contiguous(), k.contiguous(), v, cu.cpu() if cu.is_cuda else cu, max_seqlen, causal,
                                 float(scale), True)
