"""Autograd wrappers of the bandwidth-bound Llama kernels (csrc/kernels/llm_ops.cu)."""
from __future__ import annotations

import torch

from . import _lib


def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-5, residual: torch.Tensor | None = None):
    """Returns (normed, h) where h = x + residual (or x itself when residual is None); with a residual,
    h is a new tensor produced in the same pass as the normalisation."""
    out = _lib.native().rmsnorm(x, residual, weight, eps)
    return out[0], (out[1] if residual is not None else x)


def swiglu(gate_up: torch.Tensor) -> torch.Tensor:
    """silu(gate) * up for a fused [..., 2F] tensor laid out as gate | up."""
    return _lib.native().swiglu(gate_up)


def swiglu_mlp(x: torch.Tensor, w_gate_up: torch.Tensor, w_down: torch.Tensor) -> torch.Tensor:
    """``linear(swiglu(linear(x, w_gate_up)), w_down)`` as one layer: the activation and its gradient are part of
    the products beside them.  w_gate_up [2F, hidden] (gate over up) and w_down [out, F] are contiguous; their
    gradients go where those of ``linear`` go."""
    return _lib.native().swiglu_mlp(x, w_gate_up, w_down)


def rope_qkv(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, batch: int, seq: int, n_heads: int, n_kv_heads: int,
             head_dim: int) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """Rotated q and k, and v, as [batch, seq, heads, head_dim] tensors of their own from the fused
    projection [batch * seq, (n_heads + 2 * n_kv_heads) * head_dim]."""
    return tuple(_lib.native().rope_qkv(qkv, cos, sin, batch, seq, n_heads, n_kv_heads, head_dim))


class _RoPE(torch.autograd.Function):
    """In-place rotary embedding on a [T, nheads, hd] view (token pitch may exceed nheads*hd)."""

    @staticmethod
    def forward(ctx, x, cos, sin, seq):
        T, nh, hd = x.shape
        assert x.stride(2) == 1 and x.stride(1) == hd
        _lib.check(_lib.load().b200_rope(x.data_ptr(), cos.data_ptr(), sin.data_ptr(), T, nh, hd, x.stride(0), seq, 0,
                                         _lib.stream_ptr()), "rope")
        ctx.save_for_backward(cos, sin)
        ctx.seq = seq
        ctx.mark_dirty(x)
        return x

    @staticmethod
    def backward(ctx, dx):
        cos, sin = ctx.saved_tensors
        dx = dx.clone(memory_format=torch.contiguous_format)  # never rotate the caller's gradient in place
        T, nh, hd = dx.shape
        _lib.check(_lib.load().b200_rope(dx.data_ptr(), cos.data_ptr(), sin.data_ptr(), T, nh, hd, dx.stride(0),
                                         ctx.seq, 1, _lib.stream_ptr()), "rope_bwd")
        return dx, None, None, None


def rope_(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, seq: int) -> torch.Tensor:
    """Rotary embedding in place, for programs that hold q or k as [T, heads, head_dim] tensors; the model
    rotates while it splits its fused projection (``rope_qkv``)."""
    return _RoPE.apply(x, cos, sin, seq)


class _CrossEntropy(torch.autograd.Function):
    """What ``cross_entropy`` is while torch.jit.trace records it (which refuses it: it overwrites its input); otherwise it is native.
    ``assume_unit_grad``, which the native one reads as well when its backward pass runs, says whether the incoming scalar is
    taken for one; cleared, the logits' gradient is multiplied by it."""

    @staticmethod
    def forward(ctx, logits, targets):
        T, V = logits.shape
        assert logits.stride(1) == 1
        scale = 1.0 / T
        assert logits.is_cuda and logits.dtype == torch.bfloat16
        assert (targets.dtype == torch.int64 and targets.is_contiguous() and targets.numel() >= T
                and (targets.device == logits.device or targets.is_pinned()))
        loss = torch.empty(T, device=logits.device, dtype=torch.float32)
        _lib.check(_lib.load().b200_cross_entropy(logits.data_ptr(), targets.data_ptr(), loss.data_ptr(), T, V,
                                                  logits.stride(0), scale, _lib.stream_ptr()), "cross_entropy")
        ctx.save_for_backward(logits)
        ctx.mark_dirty(logits)
        # nobody differentiates through the overwritten logits: no zero-filled [T, V] gradient for them
        ctx.set_materialize_grads(False)
        return loss.mean(), logits

    @staticmethod
    def backward(ctx, dloss, dlogits_out):
        (dlogits,) = ctx.saved_tensors
        if dlogits_out is not None:
            raise RuntimeError("cross_entropy overwrites its logits with their gradient: nothing can be differentiated "
                               "through them afterwards")
        if dloss is None:   # the loss was not differentiated
            return None, None
        # dloss is 1.0 in the training loop; avoid a 1 GB multiply in that case
        if dloss.numel() == 1 and getattr(_CrossEntropy, "assume_unit_grad", True):
            return dlogits, None
        return dlogits * dloss, None


def cross_entropy(logits: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
    """Mean token cross-entropy of a [rows, classes] matrix. The logits are overwritten with the gradient of the loss in the forward
    pass (one fused kernel) and the backward pass hands them on as they are: it takes the gradient that comes in for one, so
    ``(loss / n).backward()`` gives the gradients of ``loss``. A program that scales or weights its loss clears
    ``_CrossEntropy.assume_unit_grad`` before the backward pass; the gradient is then multiplied, a pass over all logits."""
    if torch._C._get_tracing_state() is not None:
        return _CrossEntropy.apply(logits, targets)[0]
    return _lib.native().cross_entropy(logits, targets)[0]


def embedding(ids: torch.Tensor, table: torch.Tensor) -> torch.Tensor:
    return _lib.native().embedding(ids, table)


def adamw_step(p: torch.Tensor, g: torch.Tensor, m: torch.Tensor, v: torch.Tensor, master: torch.Tensor | None,
               *, lr: float, beta1: float, beta2: float, eps: float, weight_decay: float, step: int,
               grad_scale: float = 1.0, zero_grad: bool = True) -> None:
    """One fused AdamW update over flat buffers (bf16 p/g, fp32 m/v, optional fp32 master)."""
    n = p.numel()
    assert g.numel() == n and m.numel() == n and v.numel() == n and n % 8 == 0
    rc = _lib.load().b200_adamw(p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(),
                                master.data_ptr() if master is not None else None, n, lr, beta1, beta2, eps,
                                weight_decay, step, grad_scale, int(zero_grad), _lib.stream_ptr())
    _lib.check(rc, "b200_adamw")


def sumsq(x: torch.Tensor) -> torch.Tensor:
    out = torch.zeros(1, device=x.device, dtype=torch.float32)
    _lib.check(_lib.load().b200_sumsq(x.data_ptr(), x.numel(), out.data_ptr(), _lib.stream_ptr()), "sumsq")
    return out
