"""SwiGLU in the products of an MLP (the local layer and the tensor-parallel one on one rank) against 64 bits, at
the edges of tiles, of their halves and of the paths that carry it."""
import ctypes
import statistics

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


def _swiglu_product(x, w, gu, act):
    from aws_ofi_nccl_b200.ops import _lib

    ll, vp = ctypes.c_longlong, ctypes.c_void_p
    assert _lib.load().b200_gemm_swiglu(vp(x.data_ptr()), vp(w.data_ptr()), vp(gu.data_ptr()), vp(act.data_ptr()), x.shape[0], act.shape[1],
                                        x.shape[1], ll(x.shape[1]), vp(_lib.stream_ptr())) == 0


def test_gates_of_every_size_in_the_product():
    """Gates of 32 bits on both sides of the written-out form's range, beside one another in a warp and alone."""
    T, ffn = 256, 128
    gates = torch.tensor([0.0, -0.0, 1e-30, 5.0, -5.0, 79.5, -79.5, 80.0, -80.0, -84.0, -87.0, 88.5, 120.0, 1e30, 3e38], device="cuda").bfloat16()
    x = torch.zeros(T, 8, device="cuda").bfloat16()
    x[:, 0], x[:, 1] = gates.repeat(T // gates.numel() + 1)[:T], 0.75
    x[128:, 0] = gates[8]
    w = torch.zeros(2 * ffn, 8, device="cuda").bfloat16()
    w[:ffn, 0], w[ffn:, 1] = 1, 1
    gu, act = torch.empty(T, 2 * ffn, device="cuda").bfloat16(), torch.empty(T, ffn, device="cuda").bfloat16()
    _swiglu_product(x, w, gu, act)
    g = x[:, :1].double()
    want = (g * torch.sigmoid(g) * 0.75).expand(T, ffn)
    # e^80 has an argument whose product with log2(e) is rounded at 2^-17: far from a bf16 step
    assert ((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-38).all()


def test_the_activation_of_the_product_errs_by_ulps_of_32_bits():
    """Gates and ups that are exact in 32 bits. A share of E / 2^16 of the results is not the exact one rounded to bf16 where the error
    before that rounding is E ulp of 32 bits on average."""
    T = ffn = 2048
    g = torch.Generator(device="cuda").manual_seed(6)
    x, w = torch.zeros(T, 8, device="cuda").bfloat16(), torch.zeros(2 * ffn, 8, device="cuda").bfloat16()
    x[:, :2] = torch.randn(T, 2, device="cuda", generator=g) * 3
    w[:ffn, 0], w[ffn:, 1] = torch.randn(ffn, device="cuda", generator=g), torch.randn(ffn, device="cuda", generator=g)
    gu, act = torch.empty(T, 2 * ffn, device="cuda").bfloat16(), torch.empty(T, ffn, device="cuda").bfloat16()
    _swiglu_product(x, w, gu, act)
    G, U = x[:, :1].double() * w[:ffn, 0].double(), x[:, 1:2].double() * w[ffn:, 1].double()
    misses = (act != (G * torch.sigmoid(G) * U).bfloat16()).sum().item()
    assert misses / act.numel() * 2.0 ** 16 < 4


def test_large_gates_take_no_longer():
    """Timed against ordinary ones in turn; a division as a call of its own took five times as long."""
    T, ffn, K = 4096, 4096, 512
    x = torch.randn(T, K, device="cuda").bfloat16()
    w = [(torch.randn(2 * ffn, K, device="cuda") * K ** -0.5 * s).bfloat16() for s in (1, 64)]
    gu, act = torch.empty(T, 2 * ffn, device="cuda").bfloat16(), torch.empty(T, ffn, device="cuda").bfloat16()
    times = [[], []]
    for _ in range(9):
        for t, weight in zip(times, w):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                _swiglu_product(x, weight, gu, act)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
    assert statistics.median(times[1]) < 1.8 * statistics.median(times[0])


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
