"""The work a training program has this framework do, as cases that can be timed and checked.

Every case is one pass through public entry points: a decoder layer's forward and backward task, the
attention, routed-expert and delta-rule operators in both directions, the chunked output head with its
loss, the optimizer update of a layer, and a whole training step of a small model. Sizes are those of the
named presets (``models/config.py``), the packed batches those of the headline benchmark (log-normal
lengths, median 1200, at most 8192). ``exact`` restates each path in 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from shadowspill_b200.execution.resident import ResidentTrainer
from shadowspill_b200.models import autograd_ops as A
from shadowspill_b200.models.config import preset
from shadowspill_b200.models.decoder import BatchMeta, DenseLayerStage, HeadLossStage
from shadowspill_b200.ops import delta_rule
from shadowspill_b200.ops import functional as F
from shadowspill_b200.ops import moe

DEV = "cuda"
BF16 = torch.bfloat16
_HYPER = dict(lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1)


def listed() -> list[dict]:
    return [
        # the smallest whole program: one training step (forward, loss, backward, update, loss read
        # back) of the 5 M parameter preset that the plumbing tests and first runs use
        dict(name="model_step_plumbing", kind="model_step", model="llama3-plumbing", tokens=768, median=200),
        # the headline benchmark's unit of work: one layer's forward and backward task on one microbatch,
        # keeping the attention set between them, as the planner chooses for it
        dict(name="layer_llama3_8b", kind="layer", model="llama3-8b", tokens=8192, median=1200,
             variant="save_attention", first=True),
        # a layer with q/k norms on a ragged, smaller microbatch that recomputes everything and adds
        # to the gradients of the microbatch before
        dict(name="layer_qwen3_1.7b", kind="layer", model="qwen3-1.7b", tokens=1999, median=600,
             variant="recompute", first=False),
        # packed sequences of the benchmark's length mix at its head geometry
        dict(name="attention_packed", kind="attention", heads=32, kv_heads=8, width=128, tokens=8192, median=1200),
        # long-context training: sequences at the benchmark's maximum length
        dict(name="attention_long", kind="attention", heads=32, kv_heads=8, width=128, tokens=16384, median=8192),
        # the wide heads of the hybrid family (qwen35-9b), ragged total
        dict(name="attention_wide", kind="attention", heads=16, kv_heads=4, width=256, tokens=6001, median=1200),
        # the narrow heads of the 1 B preset on a short microbatch of short sequences
        dict(name="attention_narrow", kind="attention", heads=32, kv_heads=8, width=64, tokens=2048, median=300),
        # routed experts of the mixture benchmark (olmoe-7b-a1b) on one microbatch
        dict(name="experts_olmoe", kind="experts", model="olmoe-7b-a1b", tokens=8192),
        # many small experts with few rows each (qwen3moe-30b-a3b, a short microbatch)
        dict(name="experts_qwen3moe", kind="experts", model="qwen3moe-30b-a3b", tokens=1000),
        # the gated delta rule of the hybrid benchmark (qwen35-9b) on one microbatch
        dict(name="delta_rule_9b", kind="delta_rule", heads=32, kv_heads=16, tokens=8192, median=1200),
        # output head and loss over the 128 k vocabulary with both gradients, in row blocks
        dict(name="head_llama3_8b", kind="head", model="llama3-8b", tokens=4096, median=1200),
        # the optimizer's task for one layer of the headline model
        dict(name="update_llama3_8b", kind="update", model="llama3-8b"),
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["model_step", "layer", "layer", "attention", "attention", "attention", "experts", "experts",
                       "delta_rule", "head", "update"])
    if kind == "model_step":
        return dict(kind=kind, model="llama3-plumbing", tokens=_log(rng, 64, 4096), median=_log(rng, 40, 1200))
    if kind == "layer":
        return dict(kind=kind, model=rng.choice(["llama3-plumbing", "llama3-1b", "llama3-8b", "qwen3-1.7b", "qwen3-8b"]),
                    tokens=_log(rng, 64, 8100), median=_log(rng, 100, 2000),
                    variant=rng.choice(["recompute", "save_attention", "save"]), first=rng.random() < 0.5)
    if kind == "attention":
        heads, kv, width, most = rng.choice([(32, 8, 128, 16384), (16, 16, 128, 16384), (64, 8, 128, 8192),
                                             (16, 4, 256, 8192), (8, 2, 256, 8192), (32, 8, 64, 16384), (4, 2, 64, 16384)])
        return dict(kind=kind, heads=heads, kv_heads=kv, width=width, tokens=_log(rng, 64, most),
                    median=_log(rng, 100, 6000))
    if kind == "experts":
        return dict(kind=kind, model=rng.choice(["olmoe-numerical", "olmoe-7b-a1b", "qwen3moe-30b-a3b"]),
                    tokens=_log(rng, 64, 8100))
    if kind == "delta_rule":
        kv, heads = rng.choice([(6, 12), (16, 16), (16, 32), (16, 48)])
        return dict(kind=kind, heads=heads, kv_heads=kv, tokens=_log(rng, 64, 8100), median=_log(rng, 100, 2000))
    if kind == "head":
        return dict(kind=kind, model=rng.choice(["llama3-plumbing", "llama3-1b", "llama3-8b", "olmoe-7b-a1b", "qwen3-1.7b"]),
                    tokens=_log(rng, 64, 4000), median=_log(rng, 100, 2000))
    return dict(kind=kind, model=rng.choice(["llama3-plumbing", "llama3-numerical", "llama3-1b", "qwen3-1.7b", "qwen3-8b"]),
                step=rng.randint(1, 2000))


# ---------------------------------------------------------------------------- inputs
def _lengths(case) -> list[int]:
    """The packed sequence lengths of a case: log-normal as in the synthetic data of the benchmark."""
    total, median = case["tokens"], case["median"]
    rng = np.random.default_rng(total * 7919 + median)
    out = []
    while total:
        n = min(total, int(np.clip(rng.lognormal(math.log(median), 1.0), 32, 8192)))
        out.append(n)
        total -= n
    return out


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0, dtype=BF16):
    return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0.0, std, generator=g).to(dtype)


def _cu(case) -> torch.Tensor:
    return torch.tensor([0, *np.cumsum(_lengths(case)).tolist()], dtype=torch.int32, device=DEV)


def _meta(case, vocab: int, g) -> BatchMeta:
    lens, T = _lengths(case), case["tokens"]
    positions = torch.tensor(np.concatenate([np.arange(n) for n in lens]), dtype=torch.int32, device=DEV)
    tokens = torch.randint(0, vocab, (T,), generator=g, device=DEV)
    masked = (torch.arange(T, device=DEV) // 64) % 2 == 1                    # alternating loss spans
    targets = torch.where(masked, -1, torch.randint(0, vocab, (T,), generator=g, device=DEV))
    weights = (~masked).float() / float((~masked).sum())
    return BatchMeta(tokens, targets, weights, positions, _cu(case), max(lens))


def _fill(stage, P, g) -> None:
    for p in stage.params:
        if len(p.shape) == 1:
            P[p.name].copy_(1.0 + _randn(g, *p.shape, std=0.1, dtype=torch.float32))
        else:
            P[p.name].copy_(_randn(g, *p.shape, std=p.std))


def _buffers(stage):
    """Parameter and gradient buffers of a stage, laid out as the executor lays them out."""
    _, pbytes = stage.layout(BF16)
    _, gbytes = stage.layout(BF16, torch.float32)
    P = stage.views(torch.zeros(pbytes, dtype=torch.uint8, device=DEV), BF16)
    G = stage.views(torch.zeros(gbytes, dtype=torch.uint8, device=DEV), BF16, torch.float32)
    return P, G


def _attention_inputs(case, g):
    T, H, Hk, d = case["tokens"], case["heads"], case["kv_heads"], case["width"]
    return (_randn(g, T, H, d), _randn(g, T, Hk, d), _randn(g, T, Hk, d), _randn(g, T, H, d, std=0.1), _cu(case),
            max(_lengths(case)))


def _delta_inputs(case, g):
    T, H, Hk = case["tokens"], case["heads"], case["kv_heads"]
    q, k = (torch.nn.functional.normalize(_randn(g, T, Hk, 128, dtype=torch.float32), dim=-1).to(BF16) for _ in range(2))
    v, dout = _randn(g, T, H, 128), _randn(g, T, H, 128, std=0.1)
    beta = torch.sigmoid(_randn(g, T, H, dtype=torch.float32))
    rate = torch.empty(H, device=DEV).uniform_(0.02, 1.0, generator=g)
    decay = -rate * torch.nn.functional.softplus(_randn(g, T, H, dtype=torch.float32))
    return q, k, v, beta, decay, dout, _cu(case)


def _experts_inputs(case, g):
    c, T = preset(case["model"]), case["tokens"]
    h = _randn(g, T, c.d_model)
    # router scores: per-expert popularity plus token preference, so that the experts' loads differ
    logits = _randn(g, T, c.n_experts, dtype=torch.float32) + _randn(g, 1, c.n_experts, std=0.5, dtype=torch.float32)
    w13 = _randn(g, c.n_experts, 2 * c.d_expert, c.d_model, std=0.02)
    w2 = _randn(g, c.n_experts, c.d_model, c.d_expert, std=0.02)
    return h, logits, w13, w2, _randn(g, T, c.d_model, std=0.01)


def _layer_inputs(case, g):
    c = preset(case["model"])
    stage = DenseLayerStage("layer0", c)
    P, G = _buffers(stage)
    _fill(stage, P, g)
    if not case["first"]:                                   # gradients of the microbatch before
        for t in G.values():
            t.copy_(_randn(g, *t.shape, std=0.01, dtype=t.dtype))
    x, dy = _randn(g, case["tokens"], c.d_model), _randn(g, case["tokens"], c.d_model, std=0.01)
    return stage, P, G, x, dy, _meta(case, c.vocab_size, g)


def _head_inputs(case, g):
    c = preset(case["model"])
    stage = HeadLossStage("head", c)
    P, G = _buffers(stage)
    _fill(stage, P, g)
    return stage, P, G, _randn(g, case["tokens"], c.d_model), _meta(case, c.vocab_size, g)


def _update_inputs(case, g):
    stage = DenseLayerStage("layer0", preset(case["model"]))
    out, offset = [], 0
    for p in stage.params:
        n = p.numel
        grad_dtype = torch.float32 if len(p.shape) == 1 else BF16
        grad = _randn(g, n, std=1e-3, dtype=grad_dtype)
        out.append((_randn(g, n, std=0.02), grad, _randn(g, n, std=3e-4),
                    (_randn(g, n, std=1e-3, dtype=torch.float32).square() + 1e-8).to(BF16), offset))
        offset += (n + 7) // 8 * 8
    return out


def _model_inputs(case, g):
    c = preset(case["model"])
    trainer = ResidentTrainer(c, device=DEV, **_HYPER)
    for stage, P in zip(trainer.stages, trainer.P):
        _fill(stage, P, g)
    return trainer, _meta(case, c.vocab_size, g)


_INPUTS = dict(attention=_attention_inputs, delta_rule=_delta_inputs, experts=_experts_inputs, layer=_layer_inputs,
               head=_head_inputs, update=_update_inputs, model_step=_model_inputs)


def prepare(case, seed):
    return case, _INPUTS[case["kind"]](case, _gen(seed))


# ---------------------------------------------------------------------------- one pass
def run(state):
    case, inputs = state
    return _RUN[case["kind"]](case, *inputs) if case["kind"] != "update" else _run_update(case, inputs)


def _run_attention(case, q, k, v, dout, cu, longest):
    out, lse = F.attention_varlen(q, k, v, cu, longest)
    dq, dk, dv = F.attention_varlen_bwd(q, k, v, out, lse, dout, cu, longest)
    return dict(out=out, lse=lse, dq=dq, dk=dk, dv=dv)


def _run_delta(case, q, k, v, beta, decay, dout, cu):
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v, beta, decay)]
    out = delta_rule.gated_delta_rule(*leaves, cu)
    grads = torch.autograd.grad(out, leaves, dout)
    return dict(zip(("out", "dq", "dk", "dv", "dbeta", "dg"), (out.detach(), *grads)))


def _run_experts(case, h, logits, w13, w2, dout):
    c = preset(case["model"])
    G = {"w13": torch.empty_like(w13), "w2": torch.empty_like(w2)}
    h, logits = h.detach().requires_grad_(True), logits.detach().requires_grad_(True)
    out = moe.experts(h, logits, w13, w2, c.top_k, c.router_renormalize, A.GradSink(G, True))
    dh, dlogits = torch.autograd.grad(out, (h, logits), dout)
    return dict(out=out.detach(), dh=dh, dlogits=dlogits, **G)


def _run_layer(case, stage, P, G, x, dy, meta):
    y, saved = stage.forward(P, x, meta, keep=stage.SAVE_SETS[case["variant"]])
    dx = stage.backward(P, G, x, dy.clone(), meta, saved, case["first"])
    return dict(y=y, dx=dx, **{f"d_{n}": t for n, t in G.items()})


def _run_head(case, stage, P, G, x, meta):
    loss = torch.zeros(1, dtype=torch.float32, device=x.device)
    dx = stage.loss_and_backward(P, G, x, meta, loss, True)
    return dict(loss=loss, dx=dx, **{f"d_{n}": t for n, t in G.items()})


def _run_update(case, tensors):
    for p, g, m, v, offset in tensors:
        F.adamw_(p, g, m, v, step=case.get("step", 100), seed=17, offset=offset, **_HYPER)
    return [(p, m, v) for p, _, m, v, _ in tensors]


def _run_model(case, trainer, meta):
    loss = trainer.step([meta])
    grads = {f"{i}.{n}": t for i, G in enumerate(trainer.G) for n, t in G.items()}
    params = {f"{i}.{n}": t for i, P in enumerate(trainer.P) for n, t in P.items()}
    return dict(loss=loss, grads=grads, params=params)


_RUN = dict(attention=_run_attention, delta_rule=_run_delta, experts=_run_experts, layer=_run_layer, head=_run_head,
            model_step=_run_model)


# ---------------------------------------------------------------------------- work and tolerances
def _pairs(case) -> float:
    return sum(n * (n + 1) / 2 for n in _lengths(case))


def _layer_work(c, T: int, pairs: float):
    width = (c.n_heads + 2 * c.n_kv_heads) * c.head_dim
    n = c.d_model * (width + c.n_heads * c.head_dim + 3 * c.d_ff)
    return n, 6.0 * T * n + 14.0 * pairs * c.n_heads * c.head_dim


def work(case) -> dict:
    kind = case["kind"]
    c = preset(case["model"]) if "model" in case else None
    T = case.get("tokens", 0)
    if kind == "attention":
        d, H, Hk = case["width"], case["heads"], case["kv_heads"]
        # q, k, v and dout in, out and three gradients out, the log-sum-exp
        return dict(bytes=2.0 * T * d * (4 * H + 4 * Hk) + 4.0 * T * H, flops=14.0 * _pairs(case) * H * d)
    if kind == "delta_rule":
        H, Hk = case["heads"], case["kv_heads"]
        # per token and head: three products with the 128 x 128 state forward, about twice that backward
        return dict(bytes=2.0 * T * 128 * (4 * H + 4 * Hk) + 16.0 * T * H, flops=18.0 * T * H * 128 * 128)
    if kind == "experts":
        bank = 3.0 * c.n_experts * c.d_model * c.d_expert
        return dict(bytes=4.0 * bank + 2.0 * T * 4 * c.d_model + 8.0 * T * c.n_experts,
                    flops=18.0 * T * c.top_k * c.d_model * c.d_expert)
    if kind == "layer":
        n, flops = _layer_work(c, T, _pairs(case))
        return dict(bytes=(4.0 if case["first"] else 6.0) * n + 8.0 * T * c.d_model, flops=flops)
    if kind == "head":
        n = c.vocab_size * c.d_model
        return dict(bytes=4.0 * n + 4.0 * T * c.d_model, flops=6.0 * T * n)
    if kind == "update":
        return dict(bytes=14.0 * DenseLayerStage("layer0", c).parameter_count(), flops=0.0)
    n, flops = _layer_work(c, T, _pairs(case))
    head = c.vocab_size * c.d_model
    # parameters and both moments read and written, gradients written
    return dict(bytes=14.0 * (c.n_layers * n + 2 * head), flops=c.n_layers * flops + 6.0 * T * head)


def tolerance(case):
    # bf16 operands and results, 32-bit sums: about four times the distance from the 64-bit result that
    # each path shows; outputs of another correct implementation at this precision stay within it
    return {"attention": {"rel": 1.2e-2, "max": 0.4}, "delta_rule": {"rel": 2.5e-2, "max": 0.8},
            "experts": {"rel": 1.5e-2, "max": 0.4}, "layer": {"rel": 2.0e-2, "max": 0.6},
            "head": {"rel": 1.5e-2, "max": 0.5}, "update": {"rel": 1.0e-2, "max": 0.1},
            "model_step": {"rel": 3.0e-2, "max": 0.9}}[case["kind"]]


# ---------------------------------------------------------------------------- the same in 64 bits
class _Attention64(torch.autograd.Function):
    """Causal attention over packed sequences, one sequence and query head at a time."""

    @staticmethod
    def _blocks(q, k, lens):
        rep, at = q.shape[1] // k.shape[1], 0
        for n in lens:
            mask = torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1)
            for h in range(q.shape[1]):
                s = (q[at:at + n, h] @ k[at:at + n, h // rep].t()) * q.shape[2] ** -0.5
                yield slice(at, at + n), h, h // rep, s.masked_fill_(mask, -math.inf)
            at += n

    @staticmethod
    def forward(ctx, q, k, v, lens):
        out, lse = torch.empty_like(q), torch.empty(q.shape[1], q.shape[0], dtype=q.dtype, device=q.device)
        for rows, h, kh, s in _Attention64._blocks(q, k, lens):
            lse[h, rows] = torch.logsumexp(s, -1)
            out[rows, h] = torch.softmax(s, -1) @ v[rows, kh]
        ctx.save_for_backward(q, k, v, out)
        ctx.lens = lens
        ctx.mark_non_differentiable(lse)
        return out, lse

    @staticmethod
    def backward(ctx, dout, _):
        q, k, v, out = ctx.saved_tensors
        dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for rows, h, kh, s in _Attention64._blocks(q, k, ctx.lens):
            p, do = torch.softmax(s, -1), dout[rows, h]
            ds = p * (do @ v[rows, kh].t() - (do * out[rows, h]).sum(-1, keepdim=True)) * q.shape[2] ** -0.5
            dq[rows, h] = ds @ k[rows, kh]
            dk[rows, kh] += ds.t() @ q[rows, h]
            dv[rows, kh] += p.t() @ do
        return dq, dk, dv, None


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope64(x, positions, c):
    half = c.rotary_width // 2
    inv = c.rope_base ** (-torch.arange(half, dtype=torch.float64, device=x.device) * 2.0 / c.rotary_width)
    angle = positions.double()[:, None, None] * inv
    a, b = x[..., :half], x[..., half:2 * half]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), x[..., 2 * half:]], -1)


def _layer64(P, x, meta, c, lens):
    T, H, Hk, d = x.shape[0], c.n_heads, c.n_kv_heads, c.head_dim
    qkv = (_norm64(x, P["attn_norm"], c.norm_epsilon) @ P["wqkv"].t()).view(T, H + 2 * Hk, d)
    q, k, v = qkv[:, :H], qkv[:, H:H + Hk], qkv[:, H + Hk:]
    if c.qk_norm:
        q, k = _norm64(q, P["q_norm"], c.norm_epsilon), _norm64(k, P["k_norm"], c.norm_epsilon)
    att, _ = _Attention64.apply(_rope64(q, meta.positions, c), _rope64(k, meta.positions, c), v, lens)
    x = x + att.reshape(T, H * d) @ P["wo"].t()
    gate, up = (_norm64(x, P["mlp_norm"], c.norm_epsilon) @ P["w13"].t()).chunk(2, -1)
    return x + (torch.nn.functional.silu(gate) * up) @ P["w2"].t()


def _head64(P, x, meta, c):
    logits = _norm64(x, P["final_norm"], c.norm_epsilon) @ P["head"].t()
    rows = meta.targets >= 0
    picked = logits[rows].gather(1, meta.targets[rows][:, None])[:, 0]
    return (meta.weights.double()[rows] * (torch.logsumexp(logits[rows], -1) - picked)).sum()


def _leaves64(P):
    return {n: t.double().requires_grad_(True) for n, t in P.items()}


def _delta64(q, k, v, beta, decay, lens):
    """The gated delta rule, 64 tokens at a time: state' = decay state + k^T u with u solved in the chunk."""
    rep = v.shape[1] // q.shape[1]
    q, k = (t.repeat_interleave(rep, 1).transpose(0, 1) for t in (q * 128 ** -0.5, k))     # [H, T, 128]
    v, beta, decay = v.transpose(0, 1), beta.t(), decay.t()
    outs, at = [], 0
    for n in lens:
        state = torch.zeros(v.shape[0], 128, 128, dtype=v.dtype, device=v.device)
        for a in range(at, at + n, 64):
            s = slice(a, min(a + 64, at + n))
            m = s.stop - a
            G = decay[:, s].cumsum(1)
            low = torch.ones(m, m, dtype=torch.bool, device=v.device).tril()
            D = torch.exp((G[:, :, None] - G[:, None, :]).masked_fill(~low, -math.inf))
            kk = beta[:, s, None] * (k[:, s] @ k[:, s].transpose(1, 2)) * D * low.tril(-1)
            rhs = beta[:, s, None] * (v[:, s] - G.exp()[..., None] * (k[:, s] @ state))
            u = torch.linalg.solve_triangular(kk + torch.eye(m, dtype=v.dtype, device=v.device), rhs, upper=False)
            outs.append(G.exp()[..., None] * (q[:, s] @ state) + ((q[:, s] @ k[:, s].transpose(1, 2)) * D) @ u)
            last = G[:, -1:, None]
            state = last.exp() * state + (k[:, s] * (last - G[..., None]).exp()).transpose(1, 2) @ u
        at += n
    return torch.cat(outs, 1).transpose(0, 1)


def _adam64(p, g, m, v, step):
    h = _HYPER
    m = h["beta1"] * m + (1 - h["beta1"]) * g
    v = h["beta2"] * v + (1 - h["beta2"]) * g * g
    mhat, vhat = m / (1 - h["beta1"] ** step), v / (1 - h["beta2"] ** step)
    return p * (1 - h["lr"] * h["weight_decay"]) - h["lr"] * mhat / (vhat.sqrt() + h["eps"]), m, v


def exact(case, seed):
    kind = case["kind"]
    inputs = _INPUTS[kind](case, _gen(seed))
    if kind == "attention":
        q, k, v, dout = (t.double() for t in inputs[:4])
        leaves = [t.requires_grad_(True) for t in (q, k, v)]
        out, lse = _Attention64.apply(*leaves, _lengths(case))
        dq, dk, dv = torch.autograd.grad(out, leaves, dout)
        return dict(out=out, lse=lse, dq=dq, dk=dk, dv=dv)
    if kind == "delta_rule":
        leaves = [t.double().requires_grad_(True) for t in inputs[:5]]
        out = _delta64(*leaves, _lengths(case))
        grads = torch.autograd.grad(out, leaves, inputs[5].double())
        return dict(zip(("out", "dq", "dk", "dv", "dbeta", "dg"), (out, *grads)))
    if kind == "experts":
        return _experts64(preset(case["model"]), *inputs)
    if kind == "layer":
        stage, P, G, x, dy, meta = inputs
        before = {n: t.double() for n, t in G.items()}
        P, x = _leaves64(P), x.double().requires_grad_(True)
        y = _layer64(P, x, meta, stage.cfg, _lengths(case))
        dx, *grads = torch.autograd.grad(y, [x, *P.values()], dy.double())
        return dict(y=y, dx=dx, **{f"d_{n}": g if case["first"] else before[n] + g for n, g in zip(P, grads)})
    if kind == "head":
        stage, P, _, x, meta = inputs
        P, x = _leaves64(P), x.double().requires_grad_(True)
        loss = _head64(P, x, meta, stage.cfg)
        dx, *grads = torch.autograd.grad(loss, [x, *P.values()])
        return dict(loss=loss.reshape(1), dx=dx, **{f"d_{n}": g for n, g in zip(P, grads)})
    if kind == "update":
        return [_adam64(p.double(), g.double(), m.double(), v.double(), case.get("step", 100))
                for p, g, m, v, _ in inputs]
    trainer, meta = inputs
    c = trainer.cfg
    Ps = [_leaves64(P) for P in trainer.P]
    x = Ps[0]["embed"][meta.tokens]
    for P in Ps[1:-1]:
        x = _layer64(P, x, meta, c, _lengths(case))
    loss = _head64(Ps[-1], x, meta, c)
    names = [(i, n) for i, P in enumerate(Ps) for n in P]
    found = torch.autograd.grad(loss, [Ps[i][n] for i, n in names])
    grads = {f"{i}.{n}": g for (i, n), g in zip(names, found)}
    # no value for the updated parameters: the first step of a fresh optimizer moves each by its
    # gradient's sign, and the signs of gradients near zero are rounding
    return dict(loss=float(loss), grads=grads, params=None)


def _experts64(c, h, logits, w13, w2, dout):
    h, lg = h.double(), logits.double().requires_grad_(True)
    ids = torch.topk(logits, c.top_k, dim=-1).indices
    wts = (torch.softmax(lg.gather(1, ids), -1) if c.router_renormalize
           else torch.softmax(lg, -1).gather(1, ids))
    out, dh, dwts = torch.zeros_like(h), torch.zeros_like(h), torch.zeros_like(wts)
    d13, d2 = (torch.zeros(w.shape, dtype=torch.float64, device=w.device) for w in (w13, w2))
    for e in range(c.n_experts):
        rows, slot = (ids == e).nonzero(as_tuple=True)
        x = h[rows].requires_grad_(True)
        a, b = w13[e].double().requires_grad_(True), w2[e].double().requires_grad_(True)
        w = wts.detach()[rows, slot].requires_grad_(True)
        gate, up = (x @ a.t()).chunk(2, -1)
        y = (torch.nn.functional.silu(gate) * up) @ b.t() * w[:, None]
        gx, d13[e], d2[e], gw = torch.autograd.grad(y, [x, a, b, w], dout.double()[rows])
        out.index_add_(0, rows, y.detach())
        dh.index_add_(0, rows, gx)
        dwts[rows, slot] = gw
    dlogits, = torch.autograd.grad(wts, lg, dwts)
    return dict(out=out, dh=dh, dlogits=dlogits, w13=d13, w2=d2)
