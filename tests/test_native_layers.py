"""The native layers (linear, RMSNorm, SwiGLU, rotary split) as callables: what they refuse, and that
they can be traced."""
import pytest
import torch


def _layers():
    """name -> (function of fresh inputs, inputs) at small sizes."""
    from aws_ofi_nccl_b200.ops import gemm, llm

    g = torch.Generator(device="cuda").manual_seed(3)

    def rnd(*shape):
        return torch.randn(*shape, device="cuda", generator=g).bfloat16()

    ang = torch.rand(8, 16, device="cuda", generator=g)
    cos, sin = ang.cos(), ang.sin()
    w, wn = rnd(24, 32), rnd(64)
    return {
        "linear": (lambda x: gemm.linear(x, w), lambda: (rnd(5, 32),)),
        "rmsnorm": (lambda x: llm.rmsnorm(x, wn)[0], lambda: (rnd(9, 64),)),
        "rmsnorm_residual": (lambda x, r: llm.rmsnorm(x, wn, residual=r), lambda: (rnd(9, 64), rnd(9, 64))),
        "swiglu": (llm.swiglu, lambda: (rnd(7, 32),)),
        "rope_qkv": (lambda p: llm.rope_qkv(p, cos, sin, 2, 8, 2, 1, 32), lambda: (rnd(16, 128),)),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["linear", "rmsnorm", "rmsnorm_residual", "swiglu", "rope_qkv"])
def test_a_traced_layer_computes(name):
    fn, inputs = _layers()[name]
    traced = torch.jit.trace(fn, inputs(), check_trace=False)
    outs, grads = [], []
    args = [a.requires_grad_(True) for a in inputs()]   # not those that it was traced with
    for f in (fn, traced):
        out = f(*args)
        out = out if isinstance(out, tuple) else (out,)
        outs.append(out)
        grads.append(torch.autograd.grad([o.float().sum() for o in out], args))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


@pytest.mark.parametrize("call", [
    lambda llm: llm.swiglu(torch.empty(4, 0, dtype=torch.bfloat16)),
    lambda llm: llm.swiglu(torch.empty(4, 1, dtype=torch.bfloat16)),
    lambda llm: llm.rmsnorm(torch.empty(4, 0, dtype=torch.bfloat16), torch.empty(0, dtype=torch.bfloat16)),
])
def test_an_empty_row_is_an_exception(call):
    from aws_ofi_nccl_b200.ops import llm

    with pytest.raises(ZeroDivisionError):
        call(llm)
