"""Both gradients of a linear layer in one launch, against products in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
ll, vp = ctypes.c_longlong, ctypes.c_void_p


def _padded(rows, cols, g):
    """A [rows, cols] matrix whose pitch is a multiple of 16 bytes."""
    return torch.randn(rows, (cols + 7) // 8 * 8, device="cuda", generator=g).bfloat16()[:, :cols]


def _within(got, want, k, mag):
    """fp32 sums of k exact products in any order, one rounding of the output."""
    assert ((got.double() - want).abs() <= k * 2.0 ** -24 * mag + 2 * 2.0 ** -8 * want.abs()).all()


# one tile of each; ragged rows, columns and reductions; a reduction of three k-blocks and one more (eight epilogue warps and
# four); many tiles of both, the longer ones of dx or of dw, with pairs that are filled
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (5, 72, 136), (130, 264, 1000), (192, 320, 200), (193, 137, 333), (64, 2048, 4096),
                                   (2304, 1800, 515), (4096, 3000, 128)])
@pytest.mark.parametrize("w_dx,w_dw", [(128, 128), (128, 256), (192, 192), (256, 128), (256, 256)])
def test_joint_gradients(M, N, K, w_dx, w_dw):
    from aws_ofi_nccl_b200.ops import _lib

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    dy, x, w = _padded(M, N, g), _padded(M, K, g), _padded(N, K, g)
    D, X, W = dy.double(), x.double(), w.double()
    dx = torch.full((M + 1, (K + 15) // 8 * 8), 7.0, device="cuda", dtype=torch.bfloat16)
    dw = torch.full((N + 1, (K + 15) // 8 * 8), 7.0, device="cuda", dtype=torch.bfloat16)
    want = torch.zeros(N, K, device="cuda", dtype=torch.float64)
    for accumulate in (0, 1):
        rc = _lib.load().b200_linear_grads_joint(
            vp(dy.data_ptr()), vp(x.data_ptr()), vp(w.data_ptr()), vp(dx.data_ptr()), vp(dw.data_ptr()), M, N, K, ll(dy.stride(0)),
            ll(x.stride(0)), ll(w.stride(0)), ll(dx.stride(0)), ll(dw.stride(0)), accumulate, w_dx, w_dw, vp(_lib.stream_ptr()))
        assert rc == 0
        _within(dx[:M, :K], D @ W, N, D.abs() @ W.abs())
        want = want + D.T @ X
        _within(dw[:N, :K], want, M, D.T.abs() @ X.abs())
        want = dw[:N, :K].double()
    assert (dx[M:] == 7).all() and (dx[:, K:] == 7).all() and (dw[N:] == 7).all() and (dw[:, K:] == 7).all()


def _plan(M, N, K):
    from aws_ofi_nccl_b200.ops import _lib

    out = [ctypes.c_int() for _ in range(3)]
    assert _lib.load().b200_linear_grads_plan(M, N, K, *(ctypes.byref(o) for o in out)) == 0
    return out[0].value


@pytest.mark.parametrize("M,N,K,joint", [(256, 768, 256, 1), (128, 4096, 14336, 0), (4096, 4096, 4096, 1), (1000, 712, 264, 1),
                                         (157, 16520, 80, 0), (7424, 360, 80, 0), (37, 22400, 5888, 0)])
def test_linear_layer_takes_the_faster_way(M, N, K, joint):
    """One launch or two as measured; the gradients, into a tensor of their own, a bf16 and an fp32 buffer."""
    from aws_ofi_nccl_b200.ops.gemm import linear

    assert _plan(M, N, K) == joint
    g = torch.Generator(device="cuda").manual_seed(M)
    dy, x, w = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((M, N), (M, K), (N, K)))
    D, X, W = dy.double(), x.double(), w.double()
    want_dx, mag_dx, want_dw, mag_dw = D @ W, D.abs() @ W.abs(), D.T @ X, D.T.abs() @ X.abs()
    for buffer in (None, torch.bfloat16, torch.float32):
        wl = w.clone().requires_grad_(True)
        xl = x.clone().requires_grad_(True)
        if buffer is not None:
            wl.main_grad = torch.zeros(N, K, device="cuda", dtype=buffer)
        linear(xl.view(1, M, K), wl).backward(dy.view(1, M, N))
        _within(xl.grad, want_dx, N, mag_dx)
        _within(wl.grad if buffer is None else wl.main_grad, want_dw, M, mag_dw)


@pytest.mark.parametrize("M,N,K,joint", [(200, 6144, 6144, 1), (129, 8192, 8192, 1), (136, 16384, 4096, 0)])
def test_a_row_of_pair_tiles_takes_the_faster_way(M, N, K, joint):
    """129 to 256 rows over a weight that L2 does not hold."""
    test_linear_layer_takes_the_faster_way(M, N, K, joint)


@pytest.mark.parametrize("M,N,K,joint", [(144, 7488, 1280, 0), (64, 4800, 448, 0), (340, 5952, 2816, 1), (128, 2048, 1024, 1)])
def test_two_launches_overlap_where_that_is_the_faster_way(M, N, K, joint):
    """The second one comes up while the first one ends; rows and columns that single CTAs take, and a K that four warps store."""
    test_linear_layer_takes_the_faster_way(M, N, K, joint)


def test_only_one_of_the_gradients():
    from aws_ofi_nccl_b200.ops.gemm import linear

    dy, x, w = (torch.randn(*s, device="cuda").bfloat16() for s in ((300, 264), (300, 136), (264, 136)))
    both = [t.clone().requires_grad_(True) for t in (x, w)]
    want = torch.autograd.grad(linear(*both), both, dy)
    (dx,) = torch.autograd.grad(linear(both[0], w), (both[0],), dy)
    (dw,) = torch.autograd.grad(linear(x, both[1]), (both[1],), dy)
    # the same fp32 sums in tiles of other widths
    assert torch.equal(dx, want[0]) and torch.equal(dw, want[1])
