"""Work that users of the device library and of the training engine have it do on one GPU.

Every case is a plain dict with a "kind"; the sizes are those of the Llama-3-8B configuration of
``models/llama.py``, of its tiny configuration, of ``utils/bench_moe.py`` and of the tests, plus generic
odd ones. The layers are called as a training program calls them: forward, then backward.

What needs a second GPU is not here: the plugin's payload copies go to another process's device memory,
and the collectives' traffic crosses NVLink. The tensor-parallel MLP and the MoE exchange run with one
rank, where the same kernels address this GPU's own window.
"""
from __future__ import annotations

import math
import weakref

import torch
import torch.distributed as dist
import torch.nn.functional as F

from aws_ofi_nccl_b200.models.llama import Llama, LlamaConfig
from aws_ofi_nccl_b200.ops import gemm as gemm_ops
from aws_ofi_nccl_b200.ops import llm as llm_ops
from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel
from aws_ofi_nccl_b200.parallel.symm import Communicator
from aws_ofi_nccl_b200.parallel.tensor_parallel import TensorParallelMLP

DEV = "cuda"
BF16 = torch.bfloat16


def listed() -> list[dict]:
    return [
        # forward + backward of the tiny two-layer model (2 x 128 tokens): every launch is short, the
        # number of launches and the host path decide
        dict(name="llama_tiny", kind="llama", layers=2, hidden=256, heads=4, kv_heads=2, ffn=512, vocab=1024, batch=2, seq=128),
        # two decoder layers of the 8B configuration over one full sequence, with a head of an eighth of
        # the vocabulary: what most of a training step consists of
        dict(name="llama_8b_layers", kind="llama", layers=2, hidden=4096, heads=32, kv_heads=8, ffn=14336, vocab=16040, batch=1,
             seq=4096),
        # one projection of the tiny model: the smallest linear layer
        dict(name="linear_small", kind="linear", m=256, n=768, k=256),
        # the down projection of the 8B configuration on one short sequence: few rows, much weight
        dict(name="linear_short", kind="linear", m=128, n=4096, k=14336),
        # a packed batch with a ragged token count through a layer whose widths fill no tile
        dict(name="linear_ragged", kind="linear", m=1000, n=2568, k=5160),
        # fp8 forward product with the activation quantised on the way (weights are quantised once)
        dict(name="linear_fp8", kind="fp8", m=4096, n=14336, k=4096),
        # residual add + RMSNorm of the 8B configuration, forward and backward
        dict(name="norm_residual", kind="norm", t=4096, h=4096, residual=True),
        # gate / up activation of the 8B configuration
        dict(name="swiglu", kind="swiglu", t=4096, f=14336),
        # head projection with the fused softmax cross-entropy over the full vocabulary
        dict(name="head_loss", kind="head", t=2048, h=4096, v=128256),
        # optimizer update of one decoder layer's 218 M parameters, fp32 state and master copy
        dict(name="adamw_layer", kind="adamw", n=218112000, master=True),
        # dispatch and combine of utils/bench_moe.py's sizes, fp8 payload, with their gradients
        dict(name="moe_fp8", kind="moe", t=4096, h=7168, e=256, topk=8, fp8=True),
        # sequence-parallel SwiGLU MLP: all-gather -> GEMM -> SwiGLU and GEMM -> reduce-scatter kernels
        dict(name="tp_mlp", kind="tp_mlp", t=8192, h=2048, f=8192),
    ]


def _log(rng, lo: int, hi: int, step: int = 1) -> int:
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng) -> dict:
    kind = rng.choice(["llama", "linear", "linear", "fp8", "norm", "swiglu", "head", "adamw", "moe", "tp_mlp"])
    if kind == "llama":
        hd = rng.choice([64, 128])
        kv = rng.choice([1, 2, 4])
        heads = kv * rng.choice([1, 2, 4])
        return dict(kind=kind, layers=rng.randint(1, 3), hidden=hd * heads, heads=heads, kv_heads=kv, ffn=_log(rng, 256, 8192, 8),
                    vocab=_log(rng, 512, 32768, 8), batch=rng.randint(1, 3), seq=_log(rng, 32, 2048))
    if kind == "linear":
        while True:
            m, n, k = _log(rng, 16, 8192), _log(rng, 64, 28672, 8), _log(rng, 64, 14336, 8)
            if m * n * k <= 5e11:
                return dict(kind=kind, m=m, n=n, k=k)
    if kind == "fp8":
        while True:
            m, n, k = _log(rng, 256, 8192), _log(rng, 128, 28672, 8), _log(rng, 256, 14336, 16)
            if m * n * k <= 5e11:
                return dict(kind=kind, m=m, n=n, k=k)
    if kind == "norm":
        return dict(kind=kind, t=_log(rng, 1, 16384), h=_log(rng, 64, 8192, 8), residual=rng.random() < 0.7)
    if kind == "swiglu":
        return dict(kind=kind, t=_log(rng, 1, 8192), f=_log(rng, 64, 16384, 8))
    if kind == "head":
        return dict(kind=kind, t=_log(rng, 16, 2048), h=_log(rng, 256, 4096, 8), v=_log(rng, 1024, 128256, 8))
    if kind == "adamw":
        return dict(kind=kind, n=_log(rng, 1024, 218112000, 8), master=rng.random() < 0.7)
    if kind == "moe":
        e = rng.choice([8, 16, 64, 256])
        return dict(kind=kind, t=_log(rng, 16, 4096), h=_log(rng, 256, 7168, 256), e=e, topk=rng.randint(1, 8), fp8=rng.random() < 0.5)
    return dict(kind=kind, t=_log(rng, 128, 8192, 128), h=_log(rng, 256, 2048, 64), f=_log(rng, 256, 8192, 64))


# ------------------------------------------------------------------------------------------ one rank's communicator
WINDOW_BYTES = 8 << 30
_comm: list = []
_regions: list[tuple[int, int]] = []   # (begin, end) of the window's parts that living layers hold


def _communicator() -> Communicator:
    """The process's communicator: one window that all layers of the program take their parts from."""
    if not _comm:
        if not dist.is_initialized():
            dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
        torch.cuda.set_device(0)
        _comm.append(Communicator(dist.group.WORLD, WINDOW_BYTES, torch.device("cuda", 0)))
    return _comm[0]


def _take_window(nbytes: int) -> tuple[int, int]:
    nbytes = (nbytes + 4095) // 4096 * 4096
    at = 0
    for lo, hi in sorted(_regions):
        if lo - at >= nbytes:
            break
        at = max(at, hi)
    if at + nbytes > WINDOW_BYTES:
        raise RuntimeError("the communicator's window is full")
    _regions.append((at, at + nbytes))
    return at, at + nbytes


class _State:
    """What the user's program holds: plain attributes; a part of the window is given back with it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def hold(self, region):
        weakref.finalize(self, _regions.remove, region)


# ------------------------------------------------------------------------------------------ inputs
def prepare(case: dict, seed: int) -> _State:
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]

    def rnd(*shape, std=1.0):
        return (torch.randn(*shape, device=DEV, generator=g, dtype=torch.float32) * std).to(BF16)

    if kind == "llama":
        cfg = LlamaConfig(vocab_size=case["vocab"], hidden=case["hidden"], n_layers=case["layers"], n_heads=case["heads"],
                          n_kv_heads=case["kv_heads"], ffn=case["ffn"], max_seq=case["seq"])
        model = Llama(cfg, device=DEV, seed=seed)
        shape = (case["batch"], case["seq"])
        return _State(kind=kind, model=model, ids=torch.randint(0, case["vocab"], shape, device=DEV, generator=g),
                      labels=torch.randint(0, case["vocab"], shape, device=DEV, generator=g))
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return _State(kind=kind, x=rnd(m, k).requires_grad_(True), w=rnd(n, k, std=k ** -0.5).requires_grad_(True), dy=rnd(m, n))
    if kind == "fp8":
        m, n, k = case["m"], case["n"], case["k"]
        wq, ws = gemm_ops.quantize_rows_fp8(rnd(n, k, std=k ** -0.5))
        return _State(kind=kind, x=rnd(m, k), wq=wq, ws=ws)
    if kind == "norm":
        t, h, res = case["t"], case["h"], case["residual"]
        return _State(kind=kind, x=rnd(t, h).requires_grad_(True), res=rnd(t, h).requires_grad_(True) if res else None,
                      w=(1 + 0.1 * torch.randn(h, device=DEV, generator=g)).to(BF16).requires_grad_(True), dy=rnd(t, h),
                      dh=rnd(t, h) if res else None)
    if kind == "swiglu":
        t, f = case["t"], case["f"]
        return _State(kind=kind, gu=rnd(t, 2 * f).requires_grad_(True), dout=rnd(t, f))
    if kind == "head":
        t, h, v = case["t"], case["h"], case["v"]
        return _State(kind=kind, x=rnd(t, h).requires_grad_(True), w=rnd(v, h, std=0.02).requires_grad_(True),
                      targets=torch.randint(0, v, (t,), device=DEV, generator=g))
    if kind == "adamw":
        n = case["n"]
        p = rnd(n, std=0.02)
        return _State(kind=kind, p=p, g=rnd(n, std=1e-3), m=torch.randn(n, device=DEV, generator=g) * 1e-4,
                      v=torch.rand(n, device=DEV, generator=g) * 1e-6, master=p.float() if case["master"] else None, step=10)
    if kind == "moe":
        t, h, e, k = case["t"], case["h"], case["e"], case["topk"]
        region = _take_window(ExpertParallel.window_bytes(1, t, h, e, k))
        ep = ExpertParallel(_communicator(), t, h, e, k, window_offset=region[0])
        w, idx = torch.topk(torch.softmax(torch.randn(t, e, device=DEV, generator=g), -1), k, dim=-1)
        s = _State(kind=kind, ep=ep, fp8=case["fp8"], x=rnd(t, h).requires_grad_(True), idx=idx.to(torch.int32).contiguous(),
                   w=w.contiguous().requires_grad_(True), dy=rnd(t, h))
        s.hold(region)
        return s
    t, h, f = case["t"], case["h"], case["f"]
    region = _take_window(TensorParallelMLP.window_bytes(t, h))
    mlp = TensorParallelMLP(_communicator(), t, h, f, window_offset=region[0], seed=seed)
    s = _State(kind=kind, mlp=mlp, x=rnd(t, h).requires_grad_(True), dy=rnd(t, h))
    s.hold(region)
    return s


# ------------------------------------------------------------------------------------------ one pass
def run(s: _State):
    if s.kind == "llama":
        s.model.reset_grad_flags()
        loss = s.model.forward_loss(s.ids, s.labels)
        loss.backward()
        return {"loss": loss.detach(), "grads": s.model.flat_grads}
    if s.kind == "linear":
        y = gemm_ops.linear(s.x, s.w)
        dx, dw = torch.autograd.grad(y, (s.x, s.w), s.dy)
        return {"y": y.detach(), "dx": dx, "dw": dw}
    if s.kind == "fp8":
        xq, xs = gemm_ops.quantize_rows_fp8(s.x)
        return {"y": gemm_ops.gemm_fp8(xq, s.wq, xs, s.ws)}
    if s.kind == "norm":
        y, h = llm_ops.rmsnorm(s.x, s.w, residual=s.res)
        if s.res is None:
            dx, dw = torch.autograd.grad(y, (s.x, s.w), s.dy)
            return {"y": y.detach(), "dx": dx, "dw": dw}
        dx, dr, dw = torch.autograd.grad((y, h), (s.x, s.res, s.w), (s.dy, s.dh))
        return {"y": y.detach(), "h": h.detach(), "dx": dx, "dr": dr, "dw": dw}
    if s.kind == "swiglu":
        out = llm_ops.swiglu(s.gu)
        (dgu,) = torch.autograd.grad(out, (s.gu,), s.dout)
        return {"out": out.detach(), "dgu": dgu}
    if s.kind == "head":
        loss = llm_ops.cross_entropy(gemm_ops.linear(s.x, s.w), s.targets)
        dx, dw = torch.autograd.grad(loss, (s.x, s.w))
        return {"loss": loss.detach(), "dx": dx, "dw": dw}
    if s.kind == "adamw":
        s.step += 1
        llm_ops.adamw_step(s.p, s.g, s.m, s.v, s.master, lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=s.step)
        return {"p": s.p, "g": s.g, "m": s.m, "v": s.v, "master": s.master}
    if s.kind == "moe":
        rows = s.ep.dispatch(s.x, s.idx, s.w, s.fp8)
        out = s.ep.combine(rows, s.w)   # the experts between the two are GEMMs of their own
        dx, dw = torch.autograd.grad(out, (s.x, s.w), s.dy)
        return {"out": out.detach(), "dx": dx, "dw": dw}
    s.mlp.w_gate_up.grad = s.mlp.w_down.grad = None   # as optimizer.zero_grad() leaves them
    y = s.mlp(s.x)
    (dx,) = torch.autograd.grad(y, (s.x,), s.dy)
    return {"y": y.detach(), "dx": dx, "dw_gate_up": s.mlp.w_gate_up.grad, "dw_down": s.mlp.w_down.grad}


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "llama":
        T, H = case["batch"] * case["seq"], case["hidden"]
        hd = H // case["heads"]
        per_layer = H * (case["heads"] + 2 * case["kv_heads"]) * hd + H * H + 3 * H * case["ffn"]
        params = case["layers"] * per_layer + case["vocab"] * H
        # causal attention: half of the score matrix; backward has two and a half times the forward's products
        attn = case["layers"] * 3.5 * 4 * case["batch"] * case["seq"] ** 2 / 2 * H
        return {"bytes": 2 * 2 * (params + case["vocab"] * H), "flops": 6.0 * T * params + attn}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * (m * k + n * k + m * n), "flops": 6.0 * m * n * k}
    if kind == "fp8":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * m * k + n * k + 2 * m * n, "flops": 2.0 * m * n * k}
    if kind == "norm":   # x, y, dy, dx and with a residual also res, h, dh; dr is dx
        return {"bytes": 2 * case["t"] * case["h"] * (7 if case["residual"] else 4) + 4 * case["h"], "flops": 0}
    if kind == "swiglu":
        return {"bytes": 2 * case["t"] * case["f"] * 6, "flops": 0}
    if kind == "head":
        t, h, v = case["t"], case["h"], case["v"]
        return {"bytes": 4 * (t * h + v * h), "flops": 6.0 * t * h * v}
    if kind == "adamw":
        return {"bytes": case["n"] * (30 if case["master"] else 24), "flops": 0}
    if kind == "moe":   # x, dy, out, dx once; the rows and their gradients, topk times as many, written and read once each
        return {"bytes": 2 * case["t"] * case["h"] * (4 + 4 * case["topk"]), "flops": 0}
    t, h, f = case["t"], case["h"], case["f"]
    return {"bytes": 2 * (4 * t * h + 2 * 3 * h * f), "flops": 18.0 * t * h * f}


def tolerance(case: dict) -> dict:
    kind = case["kind"]
    if kind == "llama":     # a layer's rounding travels through all that follow
        return {"rel": 0.03, "max": 0.9}
    if kind == "moe" and case["fp8"]:   # e4m3 payload: a scale that differs in its last bit moves values by a step
        return {"rel": 1e-2, "max": 0.1}
    if kind == "adamw":     # fp32 state; the bf16 parameters round it
        return {"rel": 1e-4, "max": 1e-2}
    return {"rel": 1e-2, "max": 0.1}    # bf16 outputs of fp32 sums


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _exact_llama(case, s):
    cfg = s.model.cfg
    P = {k: v.detach().double().requires_grad_(True) for k, v in s.model.params.items()}
    B, S = s.ids.shape
    hd, nq, nkv = cfg.hidden // cfg.n_heads, cfg.n_heads, cfg.n_kv_heads
    inv = 1.0 / (cfg.rope_theta ** (torch.arange(0, hd, 2, device=DEV, dtype=torch.float32) / hd))
    ang = torch.outer(torch.arange(S, device=DEV, dtype=torch.float32), inv).double()
    cos, sin = ang.cos().view(1, S, 1, hd // 2), ang.sin().view(1, S, 1, hd // 2)
    mask = torch.ones(S, S, device=DEV, dtype=torch.bool).triu(1)

    def norm(x, w):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + cfg.rms_eps) * w

    def rope(t):
        a, b = t[..., : hd // 2], t[..., hd // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    h = P["embed"][s.ids]
    for i in range(cfg.n_layers):
        qkv = norm(h, P[f"l{i}.norm1"]) @ P[f"l{i}.wqkv"].T
        q = rope(qkv[..., : nq * hd].view(B, S, nq, hd)).transpose(1, 2)
        k = rope(qkv[..., nq * hd:(nq + nkv) * hd].view(B, S, nkv, hd)).transpose(1, 2).repeat_interleave(nq // nkv, 1)
        v = qkv[..., (nq + nkv) * hd:].view(B, S, nkv, hd).transpose(1, 2).repeat_interleave(nq // nkv, 1)
        p = torch.softmax((q @ k.transpose(-1, -2) * hd ** -0.5).masked_fill(mask, -math.inf), -1)
        h = h + (p @ v).transpose(1, 2).reshape(B, S, nq * hd) @ P[f"l{i}.wo"].T
        g, u = (norm(h, P[f"l{i}.norm2"]) @ P[f"l{i}.wgu"].T).split(cfg.ffn, -1)
        h = h + (F.silu(g) * u) @ P[f"l{i}.wdown"].T
    logits = norm(h, P["normf"]) @ P["lm_head"].T
    loss = F.cross_entropy(logits.view(B * S, -1), s.labels.reshape(-1))
    names = list(P)
    flat = torch.zeros(s.model.numel, device=DEV, dtype=torch.float64)
    for name, d in zip(names, torch.autograd.grad(loss, [P[n] for n in names])):
        off, _ = s.model.offsets[name]
        flat[off:off + d.numel()] = d.reshape(-1)
    return {"loss": loss.detach(), "grads": flat}


def _e4m3_rows(x, group):
    """bf16 [R, K] -> the values that e4m3 with one fp32 scale per ``group`` elements holds, in 64 bits."""
    v = x.float().view(x.shape[0], -1, group)
    scale = v.abs().amax(-1, keepdim=True).clamp_min(1e-12) * (1.0 / 448.0)
    return ((v * (1.0 / scale)).to(torch.float8_e4m3fn).double() * scale.double()).view(x.shape)


def exact(case: dict, seed: int):
    s = prepare(case, seed)
    kind = case["kind"]

    def d(t):
        return t.detach().double()

    if kind == "llama":
        return _exact_llama(case, s)
    if kind == "linear":
        return {"y": d(s.x) @ d(s.w).T, "dx": d(s.dy) @ d(s.w), "dw": d(s.dy).T @ d(s.x)}
    if kind == "fp8":
        return {"y": (_e4m3_rows(s.x, case["k"]) @ s.wq.double().T) * s.ws.double()[None, :]}
    if kind == "norm":
        x, w = d(s.x).requires_grad_(True), d(s.w).requires_grad_(True)
        h = x if s.res is None else x + d(s.res)
        y = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5) * w
        if s.res is None:
            dx, dw = torch.autograd.grad(y, (x, w), d(s.dy))
            return {"y": y.detach(), "dx": dx, "dw": dw}
        dx, dw = torch.autograd.grad((y, h), (x, w), (d(s.dy), d(s.dh)))
        return {"y": y.detach(), "h": h.detach(), "dx": dx, "dr": dx, "dw": dw}
    if kind == "swiglu":
        gu = d(s.gu).requires_grad_(True)
        gate, up = gu.split(case["f"], -1)
        out = F.silu(gate) * up
        return {"out": out.detach(), "dgu": torch.autograd.grad(out, gu, d(s.dout))[0]}
    if kind == "head":
        x, w = d(s.x), d(s.w)
        logits = x @ w.T
        lse = torch.logsumexp(logits, -1)
        loss = (lse - logits.gather(1, s.targets[:, None])[:, 0]).mean()
        dl = torch.exp(logits - lse[:, None])
        dl.scatter_add_(1, s.targets[:, None], -torch.ones_like(dl[:, :1]))
        dl /= case["t"]
        return {"loss": loss, "dx": dl @ w, "dw": dl.T @ x}
    if kind == "adamw":
        step, lr, wd = s.step + 1, 3e-4, 0.1
        g = d(s.g)
        m, v = 0.9 * d(s.m) + 0.1 * g, 0.95 * d(s.v) + 0.05 * g * g
        p = d(s.master if s.master is not None else s.p)
        p = p * (1 - lr * wd) - lr * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.95 ** step)).sqrt() + 1e-8)
        return {"p": p, "g": torch.zeros_like(g), "m": m, "v": v, "master": p if s.master is not None else None}
    if kind == "moe":
        rows = _e4m3_rows(s.x.detach(), 128) if case["fp8"] else d(s.x)
        total = d(s.w).sum(-1, keepdim=True)
        dw = (d(s.dy) * rows).sum(-1, keepdim=True).expand(-1, case["topk"])
        return {"out": rows * total, "dx": d(s.dy) * total, "dw": dw}
    f, h = case["f"], case["h"]
    wgu = d(s.mlp.w_gate_up).view(f // 32, 2, 32, h)
    wg, wu = wgu[:, 0].reshape(f, h).requires_grad_(True), wgu[:, 1].reshape(f, h).requires_grad_(True)
    x, wd_ = d(s.x).requires_grad_(True), d(s.mlp.w_down).requires_grad_(True)
    y = (F.silu(x @ wg.T) * (x @ wu.T)) @ wd_.T
    dx, dg, du, dd = torch.autograd.grad(y, (x, wg, wu, wd_), d(s.dy))
    dgu = torch.stack((dg.view(f // 32, 32, h), du.view(f // 32, 32, h)), 1).reshape(2 * f, h)
    return {"y": y.detach(), "dx": dx, "dw_gate_up": dgu, "dw_down": dd}
