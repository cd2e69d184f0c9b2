"""SwiGLU in the products of an MLP (the local layer and the tensor-parallel one on one rank) against 64 bits, at
the edges of tiles, of their halves and of the paths that carry it."""
import pytest
import torch
import torch.distributed as dist
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    from aws_ofi_nccl_b200.parallel.symm import Communicator

    own = not dist.is_initialized()
    if own:
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    c = Communicator(dist.group.WORLD, 64 << 20, torch.device("cuda", 0), wait_limit_s=2.0)
    yield c
    c.close()
    if own:
        dist.destroy_process_group()


# a bf16 result of bf16 steps: gate|up, act and d(gate)|d(up) are each rounded once (2^-9), as is the result
TOL = 4 * 2.0 ** -9


def _close(got, want):
    """In the norm of the whole and of every row and column, so that a column in the wrong place shows."""
    d = got.double() - want
    scale = want.square().mean().sqrt()
    for dim in (None, 0, 1):
        n = (lambda t: t.square().mean().sqrt()) if dim is None else (lambda t: t.square().mean(dim).sqrt())
        # a short row or column of small values has the errors of the sums that cancelled in it
        assert (n(d) <= TOL * (n(want) + (0 if dim is None else 4 * scale))).all()


def _exact(x, wg, wu, wd, dy):
    leaves = [t.detach().double().requires_grad_(True) for t in (x, wg, wu, wd)]
    X, G, U, D = leaves
    y = (F.silu(X @ G.T) * (X @ U.T)) @ D.T
    return [y.detach(), *torch.autograd.grad(y, leaves, dy.double())]


def _rnd(g, *shape, std=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * std).bfloat16()


# (tokens, ffn, hidden, out): single CTAs and a split K, where the activation is a pass of its own; one narrow tile; ragged
# tiles; columns that end inside a tile's gates; a last wave of halves; gates outside the range of the written-out division
@pytest.mark.parametrize("T,ffn,K,H,gate", [(5, 8, 24, 16, 1), (128, 1024, 8192, 512, 1), (256, 64, 64, 128, 1), (256, 128, 64, 256, 1),
                                            (300, 200, 136, 72, 1), (1000, 712, 264, 328, 1), (257, 1928, 512, 256, 1),
                                            (4096, 2056, 256, 512, 1), (300, 200, 136, 72, 60)])
def test_local_mlp(T, ffn, K, H, gate):
    from aws_ofi_nccl_b200.ops import llm

    g = torch.Generator(device="cuda").manual_seed(T + ffn)
    x, dy = _rnd(g, T, K), _rnd(g, T, H)
    wgu, wd = _rnd(g, 2 * ffn, K, std=gate * K ** -0.5), _rnd(g, H, ffn, std=ffn ** -0.5)
    want = _exact(x, wgu[:ffn], wgu[ffn:], wd, dy)
    for t in (x, wgu, wd):
        t.requires_grad_(True)
    wd.main_grad = torch.full_like(wd, 9.0)   # overwritten, then added to
    for rounds in (1, 2):
        x.grad = wgu.grad = None
        y = llm.swiglu_mlp(x.view(1, T, K), wgu, wd)
        assert y.shape == (1, T, H)
        y.backward(dy.view(1, T, H))
        _close(y.view(T, H), want[0])
        _close(x.grad, want[1])
        _close(wgu.grad, torch.cat(want[2:4]))
        _close(wd.main_grad, rounds * want[4])
    assert wd.grad_written


@pytest.mark.parametrize("T,ffn,H", [(128, 64, 64), (256, 256, 128), (384, 320, 192), (512, 1088, 256), (2048, 2624, 128)])
def test_tensor_parallel_mlp_on_one_rank(comm, T, ffn, H):
    """Single CTAs (few columns, an odd number of 128-row chunks) and CTA pairs, widths that end inside a tile."""
    from aws_ofi_nccl_b200.parallel.tensor_parallel import TensorParallelMLP, deinterleave_gate_up

    mlp = TensorParallelMLP(comm, T, H, ffn, seed=3)
    g = torch.Generator(device="cuda").manual_seed(T + ffn)
    x, dy = _rnd(g, T, H).requires_grad_(True), _rnd(g, T, H)
    wg, wu = deinterleave_gate_up(mlp.w_gate_up.detach())
    want = _exact(x, wg, wu, mlp.w_down.detach(), dy)
    y = mlp(x)
    (dx,) = torch.autograd.grad(y, (x,), dy)
    _close(y, want[0])
    _close(dx, want[1])
    for got, exact in zip(deinterleave_gate_up(mlp.w_gate_up.grad), want[2:4]):
        _close(got, exact)
    _close(mlp.w_down.grad, want[4])
