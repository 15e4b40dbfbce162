"""The workloads whose speed this package answers for: single layers and blocks of the model families, the loss head, the
optimizer step and one whole small model, each through the entry point that a training or scoring program calls.

A case is a dict of plain values.  `prepare` makes weights and inputs on the GPU from a seed, `run` makes one pass and
returns everything the caller would go on with (outputs and gradients), `work` is the traffic and arithmetic that a pass
cannot do without, `exact` the same results in 64 bits written out in plain torch.

Kinds (sizes are those of this repository's model configurations and of its benchmark):

    norm         residual add + RMSNorm, forward and backward
    attention    one GQA attention layer over a packed row (projections, QK norm, RoPE, varlen attention, output)
    scores       the attention operator alone: long rows in forward only (scoring), or with its backward; also the
                 192 / 128-wide heads of multi-head latent attention
    mlp          dense SwiGLU MLP, forward and backward
    moe          mixture-of-experts layer: router, dispatch, grouped experts, combine, forward and backward
    lm_loss      output projection + cross entropy, loss and both gradients
    gdn          gated delta net layer (projections, short convolution, delta rule, gated norm), forward and backward
    kda          Kimi delta attention operator with its gates, forward and backward
    vision       one ViT block over packed images, forward and backward
    adamw        gradient norm, clipping and AdamW update of bf16 parameters with fp32 masters
    model        a whole small dense decoder: logits, loss and all gradients
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

BF16 = torch.bfloat16
EPS = 1e-6


def listed() -> list[dict]:
    return [
        # a few dozen response tokens of a short preference pair: launches and host work are what counts here
        dict(name="norm_short", kind="norm", rows=61, hidden=2048),
        # one packed 4096-token row of the benchmark's MoE decoder (32 query / 4 key heads), four documents
        dict(name="attention_packed", kind="attention", tokens=4096, docs=4, hidden=2048, heads=32, kv_heads=4),
        # log-probabilities of a long row under a frozen 14B-shaped model: forward only, one document, odd length
        dict(name="scores_long", kind="scores", tokens=16001, docs=1, heads=40, kv_heads=8, width=128, train=False),
        # multi-head latent attention of the DeepSeek / Kimi families in training
        dict(name="scores_latent", kind="scores", tokens=4096, docs=3, heads=16, kv_heads=16, width=192, train=True),
        # dense MLP of the 8B decoder on an 8192-token row
        dict(name="mlp_dense", kind="mlp", tokens=8192, hidden=4096, inter=12288),
        # mixture of experts of the benchmark model, all 128 experts on this GPU
        dict(name="moe_layer", kind="moe", tokens=4096, hidden=2048, inter=768, experts=128, topk=8),
        # loss head of the benchmark model
        dict(name="lm_loss", kind="lm_loss", tokens=4096, hidden=2048, vocab=151936),
        # linear-attention layer of the hybrid decoders (16 key / 32 value heads of 128), packed documents of any length
        dict(name="gdn_layer", kind="gdn", tokens=4096, docs=4, hidden=2048, k_heads=16, v_heads=32),
        # per-channel-decay delta rule, a short ragged row
        dict(name="kda_ragged", kind="kda", tokens=2047, docs=3, heads=8),
        # ViT block over a handful of images of different sizes
        dict(name="vision_block", kind="vision", images=5, side=28, hidden=1152, heads=16, inter=4304),
        # optimizer step of a 60 M parameter replica (one rank's share of the 8B decoder over a node is ten times that)
        dict(name="adamw_step", kind="adamw", params=60_000_000, tensors=20),
        # a whole small decoder on a short row: what a smoke run, a draft head or a reward probe pays per step
        dict(name="model_small", kind="model", tokens=300, docs=3, layers=4, hidden=512, inter=1024, heads=8, kv_heads=2,
             vocab=32000),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["norm", "attention", "scores", "mlp", "moe", "lm_loss", "gdn", "kda", "vision", "adamw", "model"])
    if kind == "norm":
        return dict(kind=kind, rows=_log(rng, 1, 16384), hidden=8 * rng.randint(64, 1024))
    if kind == "attention":
        kv = rng.choice([1, 2, 4, 8])
        return dict(kind=kind, tokens=_log(rng, 64, 8192), docs=rng.randint(1, 8), hidden=rng.choice([1024, 2048, 4096]),
                    heads=kv * rng.choice([2, 4, 5, 8][: 4 if kv < 8 else 2]), kv_heads=kv)
    if kind == "scores":
        width = rng.choice([128, 128, 192])
        kv = rng.choice([2, 4, 8])
        return dict(kind=kind, tokens=_log(rng, 128, 8192), docs=rng.randint(1, 8), heads=kv * (1 if width == 192 else rng.choice([1, 4])),
                    kv_heads=kv, width=width, train=rng.random() < 0.6)
    if kind == "mlp":
        return dict(kind=kind, tokens=_log(rng, 16, 8192), hidden=rng.choice([1024, 2048, 4096]), inter=64 * rng.randint(16, 192))
    if kind == "moe":
        experts = rng.choice([16, 32, 64, 128])
        return dict(kind=kind, tokens=_log(rng, 32, 4096), hidden=rng.choice([1024, 2048]), inter=64 * rng.randint(4, 12),
                    experts=experts, topk=rng.choice([2, 4, 8]))
    if kind == "lm_loss":
        return dict(kind=kind, tokens=_log(rng, 64, 4096), hidden=rng.choice([1024, 2048]), vocab=8 * rng.randint(4000, 18992))
    if kind == "gdn":
        k = rng.choice([2, 4, 8, 16])
        return dict(kind=kind, tokens=_log(rng, 64, 4096), docs=rng.randint(1, 6), hidden=rng.choice([1024, 2048]), k_heads=k,
                    v_heads=k * rng.choice([1, 2]))
    if kind == "kda":
        return dict(kind=kind, tokens=_log(rng, 64, 4096), docs=rng.randint(1, 6), heads=rng.choice([2, 4, 8]))
    if kind == "vision":
        return dict(kind=kind, images=rng.randint(1, 8), side=2 * rng.randint(4, 20), hidden=1152, heads=16, inter=4304)
    if kind == "adamw":
        return dict(kind=kind, params=_log(rng, 100_000, 100_000_000), tensors=rng.randint(1, 20))
    kv = rng.choice([1, 2])
    return dict(kind=kind, tokens=_log(rng, 32, 1024), docs=rng.randint(1, 4), layers=rng.randint(1, 4), hidden=rng.choice([256, 512]),
                inter=64 * rng.randint(8, 24), heads=4 * kv, kv_heads=kv, vocab=8 * rng.randint(1000, 4000))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
class _Maker:
    """Random tensors of one seed, made on the GPU."""

    def __init__(self, seed: int):
        self.dev = torch.device("cuda")
        self.gen = torch.Generator(self.dev)
        self.gen.manual_seed(seed)
        self.host = torch.Generator()
        self.host.manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=BF16):
        return (torch.randn(*shape, generator=self.gen, device=self.dev) * std).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=self.gen, device=self.dev) * (hi - lo) + lo

    def labels(self, rows, vocab):
        lab = torch.randint(0, vocab, (rows,), generator=self.gen, device=self.dev)
        return torch.where(torch.rand(rows, generator=self.gen, device=self.dev) < 0.15, torch.full_like(lab, -100), lab)

    def bounds(self, tokens, docs):
        """Document boundaries of a packed row, int32 on the host as the data collator delivers them."""
        cuts = torch.randperm(max(tokens - 1, 1), generator=self.host)[: min(docs, tokens) - 1] + 1
        return torch.cat((torch.zeros(1, dtype=torch.long), cuts.sort().values, torch.tensor([tokens]))).to(torch.int32)

    def weights(self, module):
        """Fills a module on the GPU: matrices with 1 / sqrt(fan_in) normals, vectors with values around one (norms) or zero."""
        with torch.no_grad():
            for name, p in module.named_parameters():
                if p.dim() >= 2:
                    p.copy_(self.normal(*p.shape, std=0.5 if "conv" in name else p[0].numel() ** -0.5))
                elif name.endswith("bias"):
                    p.copy_(self.normal(*p.shape, std=0.02))
                else:
                    p.copy_(1 + self.normal(*p.shape, std=0.1))
        return module


def _positions(cu):
    return torch.cat([torch.arange(b - a) for a, b in zip(cu[:-1].tolist(), cu[1:].tolist())])


def _rope(cu, width, theta=1e6):
    ang = _positions(cu).cuda().float()[:, None] / theta ** (torch.arange(0, width, 2, device="cuda").float() / width)[None]
    return ang.cos(), ang.sin()


def _build(make, cls, *args, **kw):
    with torch.device("cuda"):
        return make.weights(cls(*args, **kw))


def _grids(case):
    """Even patch grids of `images` pictures whose sides vary around `side` patches (the same for every seed)."""
    out, gen = [], torch.Generator()
    gen.manual_seed(case["side"])
    for _ in range(case["images"]):
        h, w = (2 * max(1, int(case["side"] * (0.5 + torch.rand(1, generator=gen).item()) / 2)) for _ in range(2))
        out.append([1, h, w])
    return torch.tensor(out)


def prepare(case: dict, seed: int) -> SimpleNamespace:
    make, kind = _Maker(seed), case["kind"]
    s = SimpleNamespace(kind=kind, case=case)
    if kind == "norm":
        R, H = case["rows"], case["hidden"]
        s.w = (1 + make.normal(H, std=0.1)).requires_grad_()
        s.x, s.res = make.normal(R, H).requires_grad_(), make.normal(R, H, std=3.0).requires_grad_()
        s.dy, s.dres = make.normal(R, H, std=1e-2), make.normal(R, H, std=1e-2)
    elif kind == "attention":
        from torchturbo_b200.models.modules.transformer import Attention

        cfg = SimpleNamespace(hidden_size=case["hidden"], num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"],
                              head_dim=128, rms_norm_eps=EPS)
        s.layer = _build(make, Attention, cfg, 0, dtype=BF16)
        s.cu = make.bounds(case["tokens"], case["docs"])
        s.max_len = int((s.cu[1:] - s.cu[:-1]).max())
        s.cos, s.sin = _rope(s.cu, 128)
        s.x = make.normal(case["tokens"], case["hidden"]).requires_grad_()
        s.dy = make.normal(case["tokens"], case["hidden"], std=1e-2)
    elif kind == "scores":
        T, D = case["tokens"], case["width"]
        s.cu = make.bounds(T, case["docs"])
        s.max_len = int((s.cu[1:] - s.cu[:-1]).max())
        s.q, s.k = make.normal(T, case["heads"], D), make.normal(T, case["kv_heads"], D)
        s.v = make.normal(T, case["kv_heads"], 128)
        s.dy = make.normal(T, case["heads"], 128, std=1e-2)
        for t in (s.q, s.k, s.v):
            t.requires_grad_(case["train"])
    elif kind == "mlp":
        from torchturbo_b200.models.modules.transformer import DenseMLP

        s.layer = _build(make, DenseMLP, case["hidden"], case["inter"], dtype=BF16)
        s.x = make.normal(case["tokens"], case["hidden"]).requires_grad_()
        s.dy = make.normal(case["tokens"], case["hidden"], std=1e-2)
    elif kind == "moe":
        from torchturbo_b200.models.modules.moe import MoELayer, MoELayerConfig

        H, I, E = case["hidden"], case["inter"], case["experts"]
        s.layer = _build(make, MoELayer, MoELayerConfig(hidden_size=H, moe_ffn_hidden_size=I, num_moe_experts=E,
                                                        moe_router_topk=case["topk"], params_dtype=BF16, moe_aux_loss_coeff=1e-3))
        with torch.no_grad():
            s.layer.experts.weight1.copy_(make.normal(E * H, 2 * I, std=H ** -0.5))
            s.layer.experts.weight2.copy_(make.normal(E * I, H, std=I ** -0.5))
        s.x = make.normal(case["tokens"], H).requires_grad_()
        s.dy = make.normal(case["tokens"], H, std=1e-2)
    elif kind == "lm_loss":
        from torchturbo_b200.models.qwen3.modeling import LMHead

        s.head = _build(make, LMHead, case["hidden"], case["vocab"], bias=False, dtype=BF16)
        s.x = make.normal(1, case["tokens"], case["hidden"]).requires_grad_()
        s.labels = make.labels(case["tokens"], case["vocab"]).view(1, -1)
        s.scale = 1.0 / max(int((s.labels >= 0).sum()), 1)
    elif kind == "gdn":
        from torchturbo_b200.models.modules.mixers import GatedDeltaNet, MixerContext

        cfg = SimpleNamespace(hidden_size=case["hidden"], linear_num_key_heads=case["k_heads"], linear_num_value_heads=case["v_heads"],
                              linear_key_head_dim=128, linear_value_head_dim=128, linear_conv_kernel_dim=4, rms_norm_eps=EPS)
        s.layer = _build(make, GatedDeltaNet, cfg, 0, dtype=BF16)
        with torch.no_grad():                       # step sizes of 1e-3 .. 1e-1 and decay rates of 1 .. 16 a unit step
            dt = torch.exp(make.uniform(case["v_heads"], lo=math.log(1e-3), hi=math.log(1e-1)))
            s.layer.dt_bias.copy_(dt + torch.log(-torch.expm1(-dt)))
            s.layer.A_log.copy_(make.uniform(case["v_heads"], lo=1.0, hi=16.0).log())
        cu = make.bounds(case["tokens"], case["docs"])
        s.cu = cu
        s.ctx = MixerContext(cos=None, sin=None, cu_seqlens=cu, max_seqlen=int((cu[1:] - cu[:-1]).max()))
        s.x = make.normal(case["tokens"], case["hidden"]).requires_grad_()
        s.dy = make.normal(case["tokens"], case["hidden"], std=1e-2)
    elif kind == "kda":
        T, H = case["tokens"], case["heads"]
        s.cu = make.bounds(T, case["docs"])
        s.q, s.k, s.v = (make.normal(1, T, H * 128).requires_grad_() for _ in range(3))
        s.g, s.beta = make.normal(1, T, H, 128).requires_grad_(), make.normal(1, T, H).requires_grad_()
        s.A_log = make.uniform(H, lo=1.0, hi=16.0).log().to(BF16).requires_grad_()
        dt = torch.exp(make.uniform(H * 128, lo=math.log(1e-3), hi=math.log(1e-1)))
        s.dt_bias = (dt + torch.log(-torch.expm1(-dt))).to(BF16).requires_grad_()
        s.dy = make.normal(1, T, H, 128, std=1e-2)
    elif kind == "vision":
        from torchturbo_b200.models.qwen3_vl.modeling import VisionBlock, vision_rot_pos

        cfg = SimpleNamespace(hidden_size=case["hidden"], num_heads=case["heads"], intermediate_size=case["inter"])
        s.layer = _build(make, VisionBlock, cfg, dtype=BF16)
        grid = _grids(case)
        n = grid.prod(-1)
        s.cu = torch.cat((torch.zeros(1, dtype=torch.long), n.cumsum(0))).to(torch.int32)
        s.max_len = int(n.max())
        s.cos, s.sin = vision_rot_pos(grid, 2, case["hidden"] // case["heads"], torch.device("cuda"))
        s.x = make.normal(int(n.sum()), case["hidden"]).requires_grad_()
        s.dy = make.normal(int(n.sum()), case["hidden"], std=1e-2)
    elif kind == "adamw":
        from torchturbo_b200.engine.optimizers.fused_adamw import FusedAdamW

        s.params = [torch.nn.Parameter(make.normal(n, std=0.02)) for n in _tensor_sizes(case)]
        s.start = [p.detach().clone() for p in s.params]
        for p in s.params:
            p.grad = make.normal(*p.shape, std=1e-3)
        s.opt = FusedAdamW(s.params, lr=1e-3, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    else:
        from torchturbo_b200.models.qwen3.model import TurboQwen3ForCausalLM
        from torchturbo_b200.models.qwen3.modeling import Qwen3Config

        cfg = Qwen3Config(vocab_size=case["vocab"], hidden_size=case["hidden"], intermediate_size=case["inter"],
                          num_hidden_layers=case["layers"], num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"],
                          head_dim=128, rms_norm_eps=EPS, rope_theta=1e6, tie_word_embeddings=False)
        s.model = _build(make, TurboQwen3ForCausalLM, cfg)
        with torch.no_grad():
            s.model.model.embed_tokens.weight.copy_(make.normal(case["vocab"], case["hidden"], std=1.0))
        s.cu = make.bounds(case["tokens"], case["docs"])
        s.max_len = int((s.cu[1:] - s.cu[:-1]).max())
        s.ids = torch.randint(0, case["vocab"], (1, case["tokens"]), generator=make.gen, device="cuda")
        s.pos = _positions(s.cu).cuda().view(1, -1)
        s.labels = make.labels(case["tokens"], case["vocab"])
        s.scale = 1.0 / max(int((s.labels >= 0).sum()), 1)
    return s


def _tensor_sizes(case):
    """Sizes that fall off like a model's: a few matrices hold most parameters, many vectors hold the rest."""
    share = [1.0 / (i + 1) for i in range(case["tensors"])]
    return [max(1, int(case["params"] * w / sum(share))) for w in share]


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def _layer_grads(y, s, **more):
    named = dict(s.layer.named_parameters())
    grads = torch.autograd.grad(y, [s.x, *named.values()], s.dy)
    return dict(more, y=y, dx=grads[0], **{"d_" + n: g for n, g in zip(named, grads[1:])})


def run(s):
    from torchturbo_b200.ops import ops

    if s.kind == "norm":
        y, total = ops.rms_norm(s.x, s.w, EPS, residual=s.res)
        dx, dres, dw = torch.autograd.grad((y, total), (s.x, s.res, s.w), (s.dy, s.dres))
        return dict(y=y, total=total, dx=dx, dres=dres, dw=dw)
    if s.kind == "attention":
        return _layer_grads(s.layer(s.x, s.cos, s.sin, s.cu, s.max_len), s)
    if s.kind == "scores":
        if not s.case["train"]:
            with torch.no_grad():
                return dict(y=ops.attention(s.q, s.k, s.v, s.cu, s.max_len, causal=True))
        y = ops.attention(s.q, s.k, s.v, s.cu, s.max_len, causal=True)
        dq, dk, dv = torch.autograd.grad(y, (s.q, s.k, s.v), s.dy)
        return dict(y=y, dq=dq, dk=dk, dv=dv)
    if s.kind == "mlp":
        return _layer_grads(s.layer(s.x), s)
    if s.kind == "moe":
        y, logits = s.layer(s.x)
        s.layer.router.pop_metrics()
        return _layer_grads(y, s, logits=logits)
    if s.kind == "lm_loss":
        loss = s.head(s.x, s.labels) * s.scale
        dx, dw = torch.autograd.grad(loss, (s.x, s.head.weight))
        return dict(loss=loss, dx=dx, dw=dw)
    if s.kind == "gdn":
        return _layer_grads(s.layer(s.x, s.ctx), s)
    if s.kind == "kda":
        o, _ = ops.kda(s.q, s.k, s.v, s.g, s.beta, A_log=s.A_log, dt_bias=s.dt_bias, use_qk_l2norm_in_kernel=True,
                       use_beta_sigmoid_in_kernel=True, use_gate_in_kernel=True, cu_seqlens=s.cu)
        names = ("q", "k", "v", "g", "beta", "A_log", "dt_bias")
        grads = torch.autograd.grad(o, [getattr(s, n) for n in names], s.dy)
        return dict(y=o, **{"d" + n: g for n, g in zip(names, grads)})
    if s.kind == "vision":
        return _layer_grads(s.layer(s.x, s.cos, s.sin, s.cu, s.max_len), s)
    if s.kind == "adamw":
        norm = s.opt.grad_sq_sum().sqrt()
        s.opt.set_clip_coef((1.0 / (norm + 1e-6)).clamp(max=1.0))
        s.opt.step()
        return dict(norm=norm, params=list(s.params), masters=[s.opt.state[p]["master"] for p in s.params],
                    exp_avg=[s.opt.state[p]["exp_avg"] for p in s.params][:4],
                    exp_avg_sq=[s.opt.state[p]["exp_avg_sq"] for p in s.params][:4])
    out = s.model(input_ids=s.ids, position_ids=s.pos, cu_seq_lens_q=s.cu, max_length_q=s.max_len)
    loss = ops.cross_entropy_loss(out.logits.view(-1, out.logits.shape[-1]), s.labels) * s.scale
    named = dict(s.model.named_parameters())
    grads = torch.autograd.grad(loss, list(named.values()))
    return dict(logits=out.logits, loss=loss, **{"d_" + n: g for n, g in zip(named, grads)})


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _pairs(cu, causal):
    """Attended (query, key) pairs of a packed row."""
    n = [b - a for a, b in zip(cu[:-1].tolist(), cu[1:].tolist())]
    return sum(x * (x + 1) / 2 if causal else x * x for x in n)


def work(case: dict) -> dict:
    """Arithmetic that is a matter of the inputs' boundaries is counted for those of seed 0."""
    kind = case["kind"]
    g = torch.Generator()
    g.manual_seed(0)
    make = SimpleNamespace(host=g)
    if kind == "norm":
        R, H = case["rows"], case["hidden"]
        return dict(bytes=2 * (8 * R * H + 2 * H), flops=20 * R * H)
    if kind == "attention":
        T, H, n, m = case["tokens"], case["hidden"], case["heads"], case["kv_heads"]
        weights = H * 128 * (n + 2 * m) + 128 * n * H
        pairs = _pairs(_Maker.bounds(make, T, case["docs"]), True)
        return dict(bytes=2 * (4 * T * H + 2 * weights), flops=6 * T * weights + 3.5 * 4 * pairs * 128 * n)
    if kind == "scores":
        T, n, m, D = case["tokens"], case["heads"], case["kv_heads"], case["width"]
        io, out = T * (n * D + m * D + m * 128), T * n * 128
        fwd = 2 * _pairs(_Maker.bounds(make, T, case["docs"]), True) * n * (D + 128)
        bwd = 2 * _pairs(_Maker.bounds(make, T, case["docs"]), True) * n * (3 * D + 2 * 128)
        return dict(bytes=2 * (2 * io + 2 * out), flops=fwd + bwd) if case["train"] else dict(bytes=2 * (io + out), flops=fwd)
    if kind == "mlp":
        T, H, I = case["tokens"], case["hidden"], case["inter"]
        return dict(bytes=2 * (4 * T * H + 2 * 3 * H * I), flops=6 * T * 3 * H * I)
    if kind == "moe":
        T, H, I, E, k = (case[n] for n in ("tokens", "hidden", "inter", "experts", "topk"))
        used = min(E, T * k)
        return dict(bytes=2 * (4 * T * H + 3 * H * I * (used + E) + 2 * E * H) + 4 * T * E,
                    flops=6 * T * k * 3 * H * I + 6 * T * H * E)
    if kind == "lm_loss":
        T, H, V = case["tokens"], case["hidden"], case["vocab"]
        return dict(bytes=2 * (2 * T * H + 2 * V * H) + 8 * T, flops=6 * T * H * V)
    if kind == "gdn":
        T, H, k, v = case["tokens"], case["hidden"], case["k_heads"] * 128, case["v_heads"] * 128
        weights = H * (2 * k + 2 * v + 2 * case["v_heads"]) + v * H
        return dict(bytes=2 * (4 * T * H + 2 * weights), flops=6 * T * weights + T * case["v_heads"] * 3 * _delta_flops())
    if kind == "kda":
        T, H = case["tokens"], case["heads"]
        return dict(bytes=2 * T * H * (2 * (4 * 128 + 1) + 2 * 128), flops=T * H * 3 * _delta_flops())
    if kind == "vision":
        H, I = case["hidden"], case["inter"]
        n = _grids(case).prod(-1)
        cu = torch.cat((torch.zeros(1, dtype=torch.long), n.cumsum(0)))
        P, weights = int(n.sum()), 4 * H * H + 2 * H * I
        return dict(bytes=2 * (4 * P * H + 2 * weights), flops=6 * P * weights + 3.5 * 4 * _pairs(cu, False) * H)
    if kind == "adamw":
        return dict(bytes=28 * case["params"], flops=20 * case["params"])
    T, H, I, V, n, m = (case[x] for x in ("tokens", "hidden", "inter", "vocab", "heads", "kv_heads"))
    weights = case["layers"] * (H * 128 * (n + 2 * m) + 128 * n * H + 3 * H * I) + V * H
    pairs = _pairs(_Maker.bounds(make, T, case["docs"]), True)
    return dict(bytes=2 * (2 * weights + V * H + T * V), flops=6 * T * weights + case["layers"] * 3.5 * 4 * pairs * 128 * n)


def _delta_flops():
    """Forward operations per token and head of the chunk-wise delta rule with 64-token chunks and 128-wide heads: two
    triangular 64 x 64 score blocks, the triangular solve applied to keys and values, three products with the state and
    the masked product with the new values."""
    return 2 * (64 * 128 + 64 * 128 + 3 * 128 * 128 + 32 * 128)


def tolerance(case: dict) -> dict:
    """Largest relative error (2-norm) between two bf16 evaluations with fp32 accumulation."""
    if case["kind"] == "adamw":
        return dict(rel=4e-3)
    if case["kind"] in ("gdn", "kda", "model"):
        return dict(rel=3e-2, max=0.99)
    return dict(rel=1.5e-2, max=0.99)


# ------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------
def _leaf(t):
    return t.detach().double().requires_grad_()


def _rms64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _attn64(q, k, v, cu, causal, scale, block=4096):
    """[T, heads, D] packed attention, head by head and 4096 query rows at a time (recomputed in the backward)."""
    def piece(qh, kh, vh, first):
        sc = qh @ kh.t() * scale
        if causal:
            rows = torch.arange(first, first + qh.shape[0], device=qh.device)[:, None]
            sc = sc.masked_fill(torch.arange(kh.shape[0], device=qh.device)[None] > rows, -math.inf)
        return torch.softmax(sc, -1) @ vh

    rep, heads = q.shape[1] // k.shape[1], []
    for h in range(q.shape[1]):
        out = []
        for a, b in zip(cu[:-1].tolist(), cu[1:].tolist()):
            for r in range(a, b, block):
                e = min(b, r + block)
                last = e if causal else b
                args = (q[r:e, h], k[a:last, h // rep], v[a:last, h // rep], r - a)
                out.append(checkpoint(piece, *args, use_reentrant=False) if torch.is_grad_enabled() else piece(*args))
        heads.append(torch.cat(out))
    return torch.stack(heads, 1)


def _rotate64(x, cos, sin):
    a, b = x.chunk(2, -1)
    c, s = cos.double()[:, None], sin.double()[:, None]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _gqa64(p, x, cos, sin, cu, n, m):
    qkv = (x @ p["qkv_proj.weight"].t()).view(x.shape[0], n + 2 * m, 128)
    q = _rotate64(_rms64(qkv[:, :n], p["q_norm.weight"]), cos, sin)
    k = _rotate64(_rms64(qkv[:, n:n + m], p["k_norm.weight"]), cos, sin)
    o = _attn64(q, k, qkv[:, n + m:], cu, True, 128 ** -0.5)
    return o.reshape(x.shape[0], -1) @ p["o_proj.weight"].t()


def _swiglu64(h):
    a, b = h.chunk(2, -1)
    return F.silu(a) * b


def _delta64(q, k, v, g, beta, cu, chunk=64):
    """[T, heads, 128] (gated) delta rule by chunks; g is the log decay per head, or per head and channel."""
    vec, outs = g.dim() == 3, []
    eye = torch.eye(chunk, dtype=q.dtype, device=q.device)
    for a, b in zip(cu[:-1].tolist(), cu[1:].tolist()):
        S = torch.zeros(q.shape[1], 128, 128, dtype=q.dtype, device=q.device)
        for c in range(a, b, chunk):
            e = min(b, c + chunk)
            qc, kc, vc = (t[c:e].transpose(0, 1) for t in (q, k, v))
            G, bc = g[c:e].transpose(0, 1).cumsum(1), beta[c:e].t()[..., None]
            low = torch.ones(e - c, e - c, dtype=torch.bool, device=q.device).tril()
            if vec:
                D = (G[:, :, None] - G[:, None]).masked_fill(~low[..., None], -math.inf).exp()
                kk, qk = (torch.einsum("hik,hijk,hjk->hij", t, D, kc) for t in (kc * bc, qc))
                into, left, last = G.exp(), (G[:, -1:] - G).exp(), G[:, -1].exp()[..., None]
            else:
                D = (G[:, :, None] - G[:, None]).masked_fill(~low, -math.inf).exp()
                kk, qk = (t @ kc.transpose(1, 2) * D for t in (kc * bc, qc))
                into, left, last = G.exp()[..., None], (G[:, -1:] - G).exp()[..., None], G[:, -1].exp()[:, None, None]
            rhs = bc * vc - (kc * bc * into) @ S
            new = torch.linalg.solve_triangular(eye[: e - c, : e - c] + kk.tril(-1), rhs, upper=False, unitriangular=True)
            outs.append(((qc * into) @ S + qk @ new).transpose(0, 1))
            S = S * last + (kc * left).transpose(1, 2) @ new
    return torch.cat(outs) * 128 ** -0.5


def _unit64(x):
    return x * torch.rsqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6)


def _conv64(x, w, cu):
    """Causal depthwise convolution and SiLU inside each document; the last tap meets the current token."""
    W = w.shape[-1]
    out = [F.conv1d(F.pad(x[a:b].t(), (W - 1, 0))[None], w, groups=w.shape[0])[0].t()
           for a, b in zip(cu[:-1].tolist(), cu[1:].tolist())]
    return F.silu(torch.cat(out))


def _gdn64(p, x, case, cu):
    T, k, v = x.shape[0], case["k_heads"] * 128, case["v_heads"] * 128
    mixed = _conv64(x @ p["in_proj_qkv.weight"].t(), p["conv1d.weight"], cu)
    q, kk, vv = (t.reshape(T, -1, 128) for t in mixed.split([k, k, v], -1))
    rep = case["v_heads"] // case["k_heads"]
    q, kk = (_unit64(t).repeat_interleave(rep, 1) for t in (q, kk))
    beta = torch.sigmoid(x @ p["in_proj_b.weight"].t())
    g = -p["A_log"].exp() * F.softplus(x @ p["in_proj_a.weight"].t() + p["dt_bias"])
    o = _rms64(_delta64(q, kk, vv, g, beta, cu), p["norm.weight"])
    o = o * F.silu((x @ p["in_proj_z.weight"].t()).view(T, -1, 128))
    return o.reshape(T, v) @ p["out_proj.weight"].t()


def _moe64(p, x, case, idx):
    H, I, E, k = case["hidden"], case["inter"], case["experts"], case["topk"]
    logits = x @ p["router.weight"].t()
    prob = torch.softmax(logits.gather(1, idx), -1)
    w1, w2 = p["experts.weight1"].view(E, H, 2 * I), p["experts.weight2"].view(E, I, H)
    y = torch.zeros_like(x)
    for e in range(E):
        rows, slot = (idx == e).nonzero(as_tuple=True)
        y = y.index_add(0, rows, (_swiglu64(x[rows] @ w1[e]) * prob[rows, slot, None]) @ w2[e])
    # load balance: experts * sum over experts of (share of routed slots) * (mean softmax score)
    count = torch.bincount(idx.reshape(-1), minlength=E).double()
    aux = (torch.softmax(logits, -1).sum(0) * count).sum() * E * 1e-3 / (k * x.shape[0] ** 2)
    return y, logits, aux


def _vision64(p, x, case, cos, sin, cu):
    P, H, n = x.shape[0], case["hidden"], case["heads"]
    lin = lambda t, m: t @ p[m + ".weight"].t() + p[m + ".bias"]                                             # noqa: E731
    norm = lambda t, m: F.layer_norm(t, (H,), p[m + ".weight"], p[m + ".bias"], 1e-6)                        # noqa: E731
    q, k, v = lin(norm(x, "norm1"), "attn.qkv").view(P, 3, n, H // n).unbind(1)
    o = _attn64(_rotate64(q, cos, sin), _rotate64(k, cos, sin), v, cu, False, (H // n) ** -0.5)
    x = x + lin(o.reshape(P, H), "attn.proj")
    return x + lin(F.gelu(lin(norm(x, "norm2"), "mlp.linear_fc1"), approximate="tanh"), "mlp.linear_fc2")


def _model64(p, case, ids, pos, cu):
    h = p["model.embed_tokens.weight"][ids.view(-1)]
    inv = 1.0 / 1e6 ** (torch.arange(0, 128, 2, device=h.device).double() / 128)
    ang = pos.view(-1).double()[:, None] * inv.float().double()[None]
    for i in range(case["layers"]):
        q = {n[len(f"model.layers.{i}."):]: t for n, t in p.items() if n.startswith(f"model.layers.{i}.")}
        a = {n[len("self_attn."):]: t for n, t in q.items() if n.startswith("self_attn.")}
        h = h + _gqa64(a, _rms64(h, q["input_layernorm.weight"]), ang.cos(), ang.sin(), cu, case["heads"], case["kv_heads"])
        y = _rms64(h, q["post_attention_layernorm.weight"])
        h = h + _swiglu64(y @ q["mlp.gate_up_proj.weight"].t()) @ q["mlp.down_proj.weight"].t()
    return _rms64(h, p["model.norm.weight"]) @ p["lm_head.weight"].t()


def exact(case: dict, seed: int):
    s = prepare(case, seed)
    kind = s.kind
    if kind == "norm":
        x, res, w = _leaf(s.x), _leaf(s.res), _leaf(s.w)
        total = x + res
        y = _rms64(total, w)
        dx, dres, dw = torch.autograd.grad((y, total), (x, res, w), (s.dy.double(), s.dres.double()))
        return dict(y=y, total=total, dx=dx, dres=dres, dw=dw)
    if kind == "scores":
        q, k, v = _leaf(s.q), _leaf(s.k), _leaf(s.v)
        scale = case["width"] ** -0.5
        if not case["train"]:
            with torch.no_grad():
                return dict(y=_attn64(q, k, v, s.cu, True, scale))
        y = _attn64(q, k, v, s.cu, True, scale)
        dq, dk, dv = torch.autograd.grad(y, (q, k, v), s.dy.double())
        return dict(y=y, dq=dq, dk=dk, dv=dv)
    if kind == "lm_loss":
        x, w, lab = s.x[0].detach().double(), s.head.weight.detach().double(), s.labels[0]
        loss, dx, dw = 0.0, torch.empty_like(x), torch.zeros_like(w)
        for r in range(0, x.shape[0], 512):
            keep = (lab[r:r + 512] >= 0).double()
            at = lab[r:r + 512].clamp(min=0)[:, None]
            logp = torch.log_softmax(x[r:r + 512] @ w.t(), -1)
            loss = loss - (logp.gather(1, at)[:, 0] * keep).sum() * s.scale
            d = logp.exp_().scatter_add_(1, at, -torch.ones_like(at, dtype=torch.float64)) * (keep * s.scale)[:, None]
            dx[r:r + 512] = d @ w
            dw += d.t() @ x[r:r + 512]
        return dict(loss=loss, dx=dx.view(s.x.shape), dw=dw)
    if kind == "kda":
        names = ("q", "k", "v", "g", "beta", "A_log", "dt_bias")
        t = {n: _leaf(getattr(s, n)) for n in names}
        T, H = case["tokens"], case["heads"]
        q, k, v = (t[n].view(T, H, 128) for n in ("q", "k", "v"))
        g = -t["A_log"].exp()[:, None] * F.softplus(t["g"][0] + t["dt_bias"].view(H, 128))
        y = _delta64(_unit64(q), _unit64(k), v, g, torch.sigmoid(t["beta"][0]), s.cu)[None]
        grads = torch.autograd.grad(y, list(t.values()), s.dy.double())
        return dict(y=y, **{"d" + n: d for n, d in zip(names, grads)})
    if kind == "adamw":
        grads = [p.grad.double() for p in s.params]
        norm = torch.stack([x.square().sum() for x in grads]).sum().sqrt()
        coef = (1.0 / (norm + 1e-6)).clamp(max=1.0)
        m = [0.1 * coef * x for x in grads]
        v = [0.05 * (coef * x).square() for x in grads]
        new = [p.double() * (1 - 1e-4) - 1e-3 * (a / 0.1) / ((b / 0.05).sqrt() + 1e-8) for p, a, b in zip(s.start, m, v)]
        return dict(norm=norm, params=new, masters=new, exp_avg=m[:4], exp_avg_sq=v[:4])
    if kind == "model":
        p = {n: _leaf(t) for n, t in s.model.named_parameters()}
        logits = _model64(p, case, s.ids, s.pos, s.cu)
        loss = F.cross_entropy(logits, s.labels, ignore_index=-100, reduction="sum") * s.scale
        grads = torch.autograd.grad(loss, list(p.values()))
        return dict(logits=logits.view(1, *logits.shape), loss=loss, **{"d_" + n: g for n, g in zip(p, grads)})
    x, p = _leaf(s.x), {n: _leaf(t) for n, t in s.layer.named_parameters()}
    more, extra = {}, None
    if kind == "attention":
        y = _gqa64(p, x, s.cos, s.sin, s.cu, case["heads"], case["kv_heads"])
    elif kind == "mlp":
        y = _swiglu64(x @ p["gate_up_proj.weight"].t()) @ p["down_proj.weight"].t()
    elif kind == "moe":
        idx = (x.detach() @ p["router.weight"].detach().t()).topk(case["topk"], -1).indices
        y, logits, extra = _moe64(p, x, case, idx)
        more = dict(logits=logits)
    elif kind == "gdn":
        y = _gdn64(p, x, case, s.cu)
    else:
        y = _vision64(p, x, case, s.cos, s.sin, s.cu)
    total = (y * s.dy.double()).sum() + (extra if extra is not None else 0.0)
    grads = torch.autograd.grad(total, [x, *p.values()])
    return dict(more, y=y, dx=grads[0], **{"d_" + n: g for n, g in zip(p, grads[1:])})
