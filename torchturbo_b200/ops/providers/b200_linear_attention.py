"""Chunked (gated) delta rule for GatedDeltaNet and Kimi Delta Attention layers on B200.

The chunked evaluation splits into work that is parallel over chunks and one recurrence over chunks:

  chunk-parallel (batched GEMMs and a batched triangular solve over all `[head, chunk]` pairs at once):
      G = cumsum(g) inside the chunk,  D_ij = exp(G_i - G_j) (i >= j)
      T = (I + strict_lower(k beta k^T . D))^-1,  u = T (beta v),  w = T (beta k e^G)
      q_in = q e^G,  k_out = k e^(G_last - G),  d = e^(G_last)
  recurrence (the `delta_state` tcgen05 kernel, whose work items are 32 columns of the state of a sequence and head;
  forward and reverse):
      v_new_c = u_c - w_c S_c,        S_{c+1} = d_c (.) S_c + k_out_c^T v_new_c
  chunk-parallel again:
      o_c = q_in_c S_c + tril(q k^T . D) v_new_c

On bf16 rows with 128-wide heads the chunk-parallel work runs in fused kernels, one CTA per chunk and head (`ChunkDelta`,
csrc/delta_chunk.cu and csrc/delta_chunk_vec.cu).  Everything else (fp32 rows, other widths, boundaries that leave rows
uncovered, CPU) takes the formulation below out of torch operations:

`StateScan` is the autograd function around the recurrence: its backward is the same kernel run over the chunks in
reverse (dS_c = d_c (.) dS_{c+1} - w_c^T dv_new_c + gS_c, dv_new_c = g_c + k_out_c dS_{c+1}) followed by batched products
for the operand gradients; everything chunk-parallel is differentiated by autograd.  Without CUDA (or for head
widths other than 128) the recurrence runs as a torch loop, so the formulation is testable on CPU against the
token-by-token oracle.  Counterpart of the `chunk_gated_delta_rule` / `chunk_kda` operators of flash-linear-attention
used by the reference (ops/providers/native/gated_delta_rule.py, ops/providers/native/kda.py)."""
from __future__ import annotations

import torch

from ... import kernels as K
from ...runtime import TurboDevice
from ..base import OpImpl, OpImplKind
from ..registry import register_op
from .b200 import _aligned, _eager
from .native_linear_attention import _bounds, gdn_gates_ref, kda_gate, l2norm, repeat_key_heads

CHUNK = 64


def _kernel_ok(t: torch.Tensor, kdim: int, vdim: int) -> bool:
    return t.is_cuda and kdim == 128 and vdim == 128 and K.available()


def _scan_torch(u, w, k_out, decay, init, seq_chunks, reverse=False, add=None, s1=-1.0, s2=1.0):
    """Torch form of the recurrence (same contract as the kernel): returns (X [H, NC, C, V], states [H, NC + nseq, K, V])."""
    H, NC, C, V = u.shape
    Kd = w.shape[-1]
    nseq = len(seq_chunks)
    X = [None] * NC
    states = [None] * (NC + nseq)
    for s, (c0, n) in enumerate(seq_chunks):
        if reverse:
            S = add[:, c0 + n + s]
        else:
            S = init[:, s] if init is not None else u.new_zeros(H, Kd, V)
        states[(c0 + n if reverse else c0) + s] = S
        order = range(c0 + n - 1, c0 - 1, -1) if reverse else range(c0, c0 + n)
        for c in order:
            x = u[:, c] + s1 * (w[:, c] @ S)
            X[c] = x
            d = decay[:, c]
            S = S * (d[:, :, None] if d.dim() == 2 else d[:, None, None]) + s2 * (k_out[:, c].transpose(-1, -2) @ x)
            slot = (c if reverse else c + 1) + s
            if add is not None:
                S = S + add[:, slot]
            states[slot] = S
    return torch.stack(X, 1), torch.stack(states, 1)


class StateScan(torch.autograd.Function):
    """(u, w, k_out, decay, init) -> (v_new, states) through the `delta_state` kernel; `seq_chunks` is the host list of
    (first chunk, chunk count) per sequence and `seq_dev` the same table on the device."""

    @staticmethod
    def forward(ctx, u, w, k_out, decay, init, seq_chunks, seq_dev):
        wb, kb = w.to(torch.bfloat16).contiguous(), k_out.to(torch.bfloat16).contiguous()
        u = u.contiguous()
        decay = decay.contiguous()
        x, states = K.delta_state_scan(wb, kb, u, decay, init, None, seq_dev, reverse=False, s1=-1.0, s2=1.0,
                                       longest=max((n for _, n in seq_chunks), default=0))
        ctx.save_for_backward(wb, kb, decay, x, states, seq_dev)
        ctx.seq_chunks = seq_chunks
        ctx.has_init = init is not None
        ctx.w_dtype, ctx.k_dtype = w.dtype, k_out.dtype
        return x, states

    @staticmethod
    def backward(ctx, gx, gstates):
        wb, kb, decay, x, states, seq_dev = ctx.saved_tensors
        seq_chunks = ctx.seq_chunks
        H, NC = x.shape[:2]
        dev = x.device
        gx = gx.contiguous() if gx is not None else torch.zeros_like(x)
        gstates = gstates.contiguous() if gstates is not None else torch.zeros_like(states)
        # reverse recurrence: A = k_out, B = w
        dx, dS = K.delta_state_scan(kb, wb, gx, decay, None, gstates, seq_dev, reverse=True, s1=1.0, s2=-1.0)
        start = torch.tensor([c + s for s, (c0, n) in enumerate(seq_chunks) for c in range(c0, c0 + n)], device=dev)
        S_c = states.index_select(1, start)                     # state at the start of every chunk
        dS_n = dS.index_select(1, start + 1)                    # gradient of the state that leaves the chunk
        dw = -(dx @ S_c.transpose(-1, -2))
        dk_out = x @ dS_n.transpose(-1, -2)
        prod = dS_n * S_c
        ddecay = prod.sum((-1, -2)) if decay.dim() == 2 else prod.sum(-1)
        dinit = None
        if ctx.has_init:
            first = torch.tensor([c0 + s for s, (c0, n) in enumerate(seq_chunks)], device=dev)
            dinit = dS.index_select(1, first)
        return dx, dw.to(ctx.w_dtype), dk_out.to(ctx.k_dtype), ddecay, dinit, None, None


class ChunkDelta(torch.autograd.Function):
    """(Gated) delta rule on bf16 rows: a few kernels around the recurrence instead of batched fp32
    products over materialised chunk tensors.  v [rows, H, 128]; q, k the same or of H / rep heads; g fp32 [rows, H] or [rows, H, 128]; beta fp32 [rows, H]; init [H, nseq, 128, 128]
    or None; `tables` = (seq_chunks, chunk_rows, last slots, first slots) on the device."""

    @staticmethod
    def forward(ctx, q, k, v, g, beta, init, tables, scale, l2, want_final=True, longest=0):
        seq, chunk_rows, last, first = tables
        kw = dict(l2=l2, scale=scale)
        T, A, u, w, k_out, decay = K.delta_prep(q, k, v, g, beta, chunk_rows, **kw)
        x, states = K.delta_state_scan(w, k_out, u, decay, init, None, seq, reverse=False, s1=-1.0, s2=1.0, longest=longest)
        o = K.delta_out(q, k, v, g, beta, chunk_rows, A, x, states, **kw)
        ctx.save_for_backward(q, k, v, g, beta, T, A, w, k_out, decay, x, states, seq, chunk_rows, last, first)
        ctx.meta = (kw, init is not None)
        ctx.set_materialize_grads(False)
        return o, (states.index_select(1, last) if want_final else None)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, do, dfinal):
        q, k, v, g, beta, T, A, w, k_out, decay, x, states, seq, chunk_rows, last, first = ctx.saved_tensors
        kw, has_init = ctx.meta
        do = _aligned(do) if do is not None else torch.zeros(v.shape, dtype=v.dtype, device=v.device)
        gx, gs = K.delta_bwd_pre(q, k, v, g, beta, chunk_rows, do, A, seq.shape[0], **kw)
        if dfinal is not None:
            gs.index_copy_(1, last.long(), dfinal.contiguous())
        dx, ds = K.delta_state_scan(k_out, w, gx, decay, None, gs, seq, reverse=True, s1=1.0, s2=-1.0, zero_first=dfinal is None)
        dq, dk, dv, dg, dbeta = K.delta_bwd_post(q, k, v, g, beta, chunk_rows, do, T, x, dx, states, ds, **kw)
        return dq, dk, dv, dg, dbeta, (ds.index_select(1, first) if has_init else None), None, None, None, None, None


def _rows_for_kernel(t: torch.Tensor, R: int) -> torch.Tensor:
    """[B, T, H, 128] -> [rows, H, 128]; copied only where a row would not start on a 16-byte boundary."""
    t = t.reshape(R, *t.shape[2:])
    if t.stride(2) != 1 or t.stride(0) % 8 or t.stride(1) % 8 or t.data_ptr() % 16:
        t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _chunk_tables(segs, C: int, device):
    """Device tables of the chunked layout, sent in one copy: per sequence (first chunk, chunks), per chunk (first row, rows,
    sequence), and the state slots behind the last / before the first chunk of every sequence."""
    seq, rows, last, first, c = [], [], [], [], 0
    for s, (base, a, b) in enumerate(segs):
        n = (b - a + C - 1) // C
        seq += [c, n]
        for r in range(a, b, C):
            rows += [base + r, min(C, b - r), s]
        first.append(c + s)
        c += n
        last.append(c + s)
    nseq = len(segs)
    host = torch.tensor(seq + rows + last + first, dtype=torch.int32).pin_memory()
    dev = host.to(device, non_blocking=True)
    seq_d, rows_d, slots_d = dev.split([2 * nseq, 3 * c, 2 * nseq])
    last_d, first_d = slots_d.split(nseq)
    return seq_d.view(nseq, 2), rows_d.view(c, 3), last_d, first_d


def _fused_usable(q, k, v, g, beta, segs, scale, rep: int = 1) -> bool:
    """The fused kernels take bf16 q / k / v of 128-wide heads and sequences that cover every row (fp32 rows would lose
    mantissa bits as tensor-core operands; they keep the batched fp32 products)."""
    R = q.shape[0] * q.shape[1]
    return (_kernel_ok(q, q.shape[-1], v.shape[-1]) and all(t.dtype == torch.bfloat16 and t.is_cuda for t in (q, k, v))
            and k.shape == q.shape and v.shape == (*q.shape[:2], q.shape[2] * rep, q.shape[3])
            and (g.shape == v.shape[:3] or (rep == 1 and g.shape == v.shape))
            and beta.shape == v.shape[:3] and scale != 0
            and 0 < v.shape[2] <= 65535 and R > 0 and sum(b - a for _, a, b in segs) == R
            and all(0 <= a <= b <= q.shape[1] for _, a, b in segs))


def _layout(segs, T_total: int, C: int, device):
    """Gather / scatter indices between packed tokens and the zero-padded `[chunk, C]` layout."""
    gather, seq_chunks, inv = [], [], torch.full((T_total,), -1, dtype=torch.long)
    c = 0
    for base, a, b in segs:
        L = b - a
        n = (L + C - 1) // C
        idx = torch.full((n * C,), T_total, dtype=torch.long)         # padding reads the appended zero row
        idx[:L] = torch.arange(base + a, base + b)
        inv[base + a: base + b] = c * C + torch.arange(L)
        gather.append(idx)
        seq_chunks.append((c, n))
        c += n
    gather = torch.cat(gather) if gather else torch.zeros(0, dtype=torch.long)
    return gather.to(device), inv.to(device), seq_chunks, c


def _channel_decay_products(kb, qc, kc, G, head_slab: int = 8, sub: int = 16):
    """`sum_k x[i, k] kc[j, k] exp(G[i, k] - G[j, k])` on `i >= j` (zero above the diagonal) for `x` in (kb, qc), with
    per-channel cumulative log decays `G [H, NC, C, K]` (non-increasing along C).

    The chunk is cut into sub-chunks of `sub` rows.  Between different sub-chunks the decay factorises around the first
    row `r` of the later one, `exp(G_i - G_r) exp(G_r - G_j)`, with both exponents non-positive, so those blocks are
    plain matrix products; only the `sub x sub` diagonal blocks materialise pairwise decays (`[.., sub, sub, K]`, a
    sixteenth of the `[.., C, C, K]` tensor per block row), a few heads at a time."""
    H, NC, C, Kd = G.shape
    nsb = C // sub
    x = torch.stack((kb, qc))                                              # [2, H, NC, C, K]
    rows = []
    tril = torch.ones(sub, sub, dtype=torch.bool, device=G.device).tril()
    for a in range(nsb):
        ra = slice(a * sub, (a + 1) * sub)
        Ga = G[:, :, ra]                                                    # [H, NC, sub, K]
        parts = []
        if a > 0:
            ref = Ga[:, :, :1]                                              # first row of this sub-chunk
            left = x[:, :, :, ra] * (Ga - ref).exp()
            right = kc[:, :, : a * sub] * (ref - G[:, :, : a * sub]).exp()
            parts.append(left @ right.transpose(-1, -2))                    # [2, H, NC, sub, a * sub]
        diag = []
        for h0 in range(0, H, head_slab):
            sl = slice(h0, h0 + head_slab)
            Dm = (Ga[sl, :, :, None, :] - Ga[sl, :, None, :, :]).masked_fill(~tril[None, None, :, :, None], -float("inf")).exp()
            diag.append(torch.einsum("xhnik,hnijk,hnjk->xhnij", x[:, sl, :, ra], Dm, kc[sl, :, ra]))
        parts.append(torch.cat(diag, 1))
        if a + 1 < nsb:
            parts.append(x.new_zeros(2, H, NC, sub, C - (a + 1) * sub))
        rows.append(torch.cat(parts, -1))
    out = torch.cat(rows, -2)                                               # [2, H, NC, C, C]
    return out[0], out[1]


def chunk_delta_rule_batched(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False, cu_seqlens=None,
                             use_qk_l2norm=False, head_slab: int = 8, heads_per_key: int = 1):
    """q, k: [B, T, H / heads_per_key, K]; v: [B, T, H, V]; g: [B, T, H] (scalar log decay) or [B, T, H, K]; beta: [B, T, H].
    Returns (o [B, T, H, V] in v's dtype, final state [N, H, K, V] fp32 or None)."""
    B, T, H, Kd = q.shape
    H *= heads_per_key
    V = v.shape[-1]
    dt = v.dtype
    dev = q.device
    C = CHUNK
    scale = Kd ** -0.5 if scale is None else scale
    if cu_seqlens is not None and B != 1:
        raise ValueError("packed delta rule expects a single row")
    segs = [(0, a, b) for a, b in _bounds(cu_seqlens, T)] if cu_seqlens is not None else [(r * T, 0, T) for r in range(B)]
    if _fused_usable(q, k, v, g, beta, segs, scale, heads_per_key):
        R = B * T
        tables = _chunk_tables(segs, C, dev)
        init = initial_state.float().transpose(0, 1).contiguous() if initial_state is not None else None
        o, final = ChunkDelta.apply(*(_rows_for_kernel(t, R) for t in (q, k, v)), g.float().reshape(R, *g.shape[2:]).contiguous(),
                                    beta.float().reshape(R, H).contiguous(), init, tables, float(scale), bool(use_qk_l2norm), bool(output_final_state),
                                    max((b - a + C - 1 for _, a, b in segs), default=0) // C)
        return o.view(B, T, H, V), (final.transpose(0, 1).contiguous() if output_final_state else None)
    q, k = (repeat_key_heads(t, heads_per_key) for t in (q, k))
    qf, kf, vf, gf, bf = (t.float() for t in (q, k, v, g, beta))
    if use_qk_l2norm:
        qf, kf = l2norm(qf), l2norm(kf)
    vec = gf.dim() == 4
    # sequences that are whole chunks and tile the rows need no gather: the chunk layout is a view of the packed rows
    aligned = all((b - a) % C == 0 for _, a, b in segs) and sum(b - a for _, a, b in segs) == B * T
    if aligned:
        seq_chunks, NC = [], 0
        for _, a, b in segs:
            seq_chunks.append((NC, (b - a) // C))
            NC += (b - a) // C
        gather = inv = None
    else:
        gather, inv, seq_chunks, NC = _layout(segs, B * T, C, dev)

    def to_chunks(x):                                   # [B, T, H, ...] -> [H, NC, C, ...]
        flat = x.reshape(B * T, *x.shape[2:])
        if not aligned:
            flat = torch.cat((flat, flat.new_zeros(1, *flat.shape[1:])), 0).index_select(0, gather)
        return flat.reshape(NC, C, *flat.shape[1:]).movedim(2, 0)

    qc, kc, vc = to_chunks(qf) * scale, to_chunks(kf), to_chunks(vf)            # [H, NC, C, K|V]
    bc = to_chunks(bf.unsqueeze(-1)).squeeze(-1)                                # [H, NC, C]
    G = (to_chunks(gf) if vec else to_chunks(gf.unsqueeze(-1)).squeeze(-1)).cumsum(2)
    eye = torch.eye(C, dtype=torch.float32, device=dev)
    low = torch.ones(C, C, dtype=torch.bool, device=dev).tril(-1)
    lowd = torch.ones(C, C, dtype=torch.bool, device=dev).tril()
    kb = kc * bc[..., None]
    if vec:
        kk, qk = _channel_decay_products(kb, qc, kc, G, head_slab)
        eG = G.exp()
        k_in, q_in = kb * eG, qc * eG
        k_out = kc * (G[:, :, -1:, :] - G).exp()
        decay = G[:, :, -1].exp()                                               # [H, NC, K]
    else:
        Dm = (G[..., :, None] - G[..., None, :]).masked_fill(~lowd, -float("inf")).exp()
        kk = (kb @ kc.transpose(-1, -2)) * Dm
        qk = (qc @ kc.transpose(-1, -2)) * Dm
        eG = G.exp()[..., None]
        k_in, q_in = kb * eG, qc * eG
        k_out = kc * (G[..., -1:] - G).exp()[..., None]
        decay = G[..., -1].exp()                                                # [H, NC]
    Tm = torch.linalg.solve_triangular(eye + kk.masked_fill(~low, 0.0), eye.expand(H, NC, C, C), upper=False)
    u = Tm @ (vc * bc[..., None])
    w = Tm @ k_in
    init = None
    if initial_state is not None:
        init = initial_state.float().transpose(0, 1).contiguous()               # [H, N, K, V]
    if _kernel_ok(q, Kd, V):
        seq_dev = torch.tensor(seq_chunks, dtype=torch.int32).pin_memory().to(dev, non_blocking=True)
        v_new, states = StateScan.apply(u, w, k_out, decay, init, seq_chunks, seq_dev)
    else:
        v_new, states = _scan_torch(u, w, k_out, decay, init, seq_chunks)
    start = torch.tensor([c + s for s, (c0, n) in enumerate(seq_chunks) for c in range(c0, c0 + n)], device=dev)
    S_c = states.index_select(1, start)
    o = q_in @ S_c + qk.masked_fill(~lowd, 0.0) @ v_new                          # [H, NC, C, V]
    o = o.movedim(0, 2).reshape(NC * C, H, V)
    if aligned:
        o = o.reshape(B, T, H, V)
    else:
        covered = sum(b - a for _, a, b in segs) == B * T
        o = o.index_select(0, inv.clamp_min(0)).reshape(B, T, H, V)
        if not covered:                                                         # rows past the last boundary read as zero
            o = o * (inv >= 0).reshape(B, T, 1, 1)
    final = None
    if output_final_state:
        last = torch.tensor([c0 + n + s for s, (c0, n) in enumerate(seq_chunks)], device=dev)
        final = states.index_select(1, last).transpose(0, 1).contiguous()
    return o.to(dt), final


class KDAGate(torch.autograd.Function):
    """`kda_gate` on bf16 rows of 128-wide heads: one kernel forward, one and a column sum backward."""

    @staticmethod
    def forward(ctx, g, A_log, dt_bias, lower_bound):
        ctx.save_for_backward(g, A_log, dt_bias)
        ctx.lower_bound = lower_bound
        return K.kda_gate_fwd(g, A_log, dt_bias, lower_bound)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dd):
        g, A_log, dt_bias = ctx.saved_tensors
        dg, ddt, da = K.kda_gate_bwd(dd.contiguous(), g, A_log, dt_bias, ctx.lower_bound)
        return dg, da.sum(-1).to(A_log.dtype), (ddt.to(dt_bias.dtype) if dt_bias is not None else None), None


def _gate(g, A_log, dt_bias, lower_bound):
    H, Kd = g.shape[-2:]
    plain = (torch.bfloat16, torch.float32)
    if (_kernel_ok(g, Kd, 128) and (lower_bound is None or isinstance(lower_bound, (int, float)))
            and g.dtype == torch.bfloat16 and A_log.is_cuda and A_log.shape == (H,) and A_log.dtype in plain
            and (dt_bias is None or (dt_bias.is_cuda and dt_bias.numel() == H * Kd and dt_bias.dtype in plain))):
        dt = dt_bias.reshape(H * Kd).contiguous() if dt_bias is not None else None
        return KDAGate.apply(g.reshape(-1, H, Kd).contiguous(), A_log.contiguous(), dt, lower_bound).view(g.shape)
    return kda_gate(g, A_log, dt_bias, lower_bound)


class GDNGatesFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, a, b, A_log, dt_bias):
        g, beta = K.gdn_gate_fwd(a, b, A_log, dt_bias)
        ctx.save_for_backward(a, b, A_log, dt_bias, beta)
        return g, beta

    @staticmethod
    def backward(ctx, dg, dbeta):
        a, b, A_log, dt_bias, beta = ctx.saved_tensors
        if torch.is_grad_enabled():              # a graph of the gradient is wanted: by way of the separate operations
            needs = ctx.needs_input_grad
            given = [t for t, n in zip((a, b, A_log, dt_bias), needs) if n]
            grads = iter(torch.autograd.grad(gdn_gates_ref(a, b, A_log, dt_bias), given, (dg, dbeta), create_graph=True, allow_unused=True))
            return tuple(next(grads) if n else None for n in needs)
        same = A_log.dtype == dt_bias.dtype
        da, db, dA, dd = K.gdn_gate_bwd(dg.contiguous(), dbeta.contiguous(), a, A_log, dt_bias, beta, A_log.dtype if same else torch.float32)
        return da, db, dA.to(A_log.dtype), dd.to(dt_bias.dtype)


def _register(op_name: str, impl_name: str):
    return register_op(op_name=op_name, impl_name=impl_name, kind=OpImplKind.CUSTOM, priority=100, devices=(TurboDevice.CUDA,))


@_register("gdn_gates", "b200_gdn_gates")
class B200GDNGates(OpImpl):
    """One launch forward and two backward.  Projections may be columns of a wider matrix, but next to one another: `a` and `b` as
    sequence parallelism leaves them, alternating in memory, take torch operations."""

    def available(self) -> bool:
        return K.available()

    def __call__(self, a, b, A_log, dt_bias):
        plain, H = (torch.bfloat16, torch.float32), a.shape[-1]
        if not (a.dim() == 2 and b.shape == a.shape and H > 0 and all(t.is_cuda and t.dtype == torch.bfloat16 and t.stride(1) == 1 for t in (a, b))
                and all(t.is_cuda and t.dtype in plain and t.shape == (H,) for t in (A_log, dt_bias)) and _eager(a, b, A_log, dt_bias)):
            return gdn_gates_ref(a, b, A_log, dt_bias)
        return GDNGatesFn.apply(a, b, A_log.contiguous(), dt_bias.contiguous())


@_register("gated_delta_rule", "b200_chunk_gated_delta_rule")
class B200GatedDeltaRule(OpImpl):
    def available(self) -> bool:
        return K.available()

    def __call__(self, q, k, v, g, beta, *, scale=None, initial_state=None, output_final_state=False,
                 use_qk_l2norm_in_kernel=False, cu_seqlens=None, packed_params=None, chunk_size=64, heads_per_key=1, **_):
        if packed_params is not None:
            if cu_seqlens is not None:
                raise ValueError("pass either cu_seqlens or packed_params, not both")
            cu_seqlens = packed_params.cu_seqlens
        return chunk_delta_rule_batched(q, k, v, g, beta, scale, initial_state, output_final_state, cu_seqlens,
                                        use_qk_l2norm_in_kernel, heads_per_key=heads_per_key)


@_register("kda", "b200_chunk_kda")
class B200KDA(OpImpl):
    """q, k: [B, T, H*K]; v: [B, T, H*V]; g: [B, T, H, K]; beta: [B, T, H].  Returns `[B, T, H, V]`."""

    def available(self) -> bool:
        return K.available()

    def __call__(self, q, k, v, g, beta, *, A_log=None, dt_bias=None, scale=None, initial_state=None,
                 output_final_state=False, use_qk_l2norm_in_kernel=False, use_beta_sigmoid_in_kernel=True,
                 use_gate_in_kernel=False, safe_gate=False, lower_bound=None, cu_seqlens=None, chunk_size=64):
        Kd = g.shape[-1]
        H = beta.shape[-1]
        if q.dim() == 3:
            q, k = q.unflatten(-1, (H, Kd)), k.unflatten(-1, (H, Kd))
        if v.dim() == 3:
            v = v.unflatten(-1, (H, -1))
        if use_gate_in_kernel:
            if A_log is None:
                raise ValueError("use_gate_in_kernel needs A_log")
            g = _gate(g, A_log, dt_bias, lower_bound if safe_gate else None)
        if use_beta_sigmoid_in_kernel:
            beta = torch.sigmoid(beta.float())
        return chunk_delta_rule_batched(q, k, v, g, beta, scale, initial_state, output_final_state, cu_seqlens,
                                        use_qk_l2norm_in_kernel)


__all__ = ["B200GatedDeltaRule", "B200KDA", "StateScan", "chunk_delta_rule_batched"]
