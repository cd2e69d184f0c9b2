"""The bandwidth kernels at the sizes where their work splits change: widths around the threads-per-row
steps, token counts around a CTA's rows, vector counts around an unrolled pass."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _within(got, ref, rel, abs_):
    """|got - ref| <= rel * |ref| + abs_, element by element, against 64 bits."""
    err = (got.double() - ref).abs()
    assert (err <= rel * ref.abs() + abs_).all(), (err - rel * ref.abs()).max().item()


BF = 2.0 ** -8   # one rounding to bf16, as a relative error (half an ulp is 2^-9; a tie in the fp32 value may add one)


@pytest.mark.parametrize("T,H", [(1, 8), (9, 256), (7, 264), (17, 520), (5, 1032), (600, 2048), (3, 2056), (299, 4096), (4, 4104),
                                 (5, 6152), (301, 8192)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm(T, H, with_res):
    from aws_ofi_nccl_b200.ops import llm

    g = torch.Generator(device="cuda").manual_seed(T * 31 + H)
    x, r, dy, dh = (torch.randn(T, H, device="cuda", generator=g).bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    x.requires_grad_(True), r.requires_grad_(True), w.requires_grad_(True)
    y, h = llm.rmsnorm(x, w, 1e-5, residual=r if with_res else None)
    got = torch.autograd.grad((y, h) if with_res else y, (x, w) + ((r,) if with_res else ()), (dy, dh) if with_res else dy)
    hq = h.detach().double()   # the kernel normalises the rounded sum
    rstd = torch.rsqrt(hq.pow(2).mean(-1, keepdim=True) + 1e-5)
    W, D = w.detach().double(), dy.double()
    _within(y.detach(), hq * rstd * W, 2 * BF, 1e-6)
    gw = D * W
    dx = rstd * (gw - hq * rstd ** 2 * (gw * hq).mean(-1, keepdim=True)) + (dh.double() if with_res else 0)
    _within(got[0], dx, 2 * BF, 1e-4)
    terms = D * hq * rstd
    _within(got[1], terms.sum(0), 2 * BF, 2.0 ** -20 * math.sqrt(T) * terms.abs().max().item() + 1e-6)
    if with_res:
        assert torch.equal(got[0], got[2])


# more groups of rows than CTAs: eight to one rows in a group, ragged last groups and widths, one group and a row more than the CTAs take at once
@pytest.mark.parametrize("T,H", [(20001, 8), (3553, 64), (3553, 256), (7003, 264), (1777, 520), (889, 2048), (445, 2056), (4001, 4096), (445, 4104),
                                 (1201, 6144), (445, 6152), (1800, 8192)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_of_many_rows(T, H, with_res):
    from aws_ofi_nccl_b200.ops import _lib

    test_rmsnorm(T, H, with_res)
    assert _lib.read_status() == 0


# rows that come through a ring of shared memory, forward, backward or both: eight to one rows in a group, ragged last groups and widths, every layout
# of a row, the fewest rows that take it, several rounds of the ring
@pytest.mark.parametrize("T,H,with_res,forward,backward", [
    (23441, 256, 0, 1, 0), (22729, 264, 0, 1, 0), (63551, 264, 1, 1, 0), (11721, 512, 0, 1, 0), (4003, 512, 1, 1, 0), (65537, 512, 0, 1, 1),
    (11539, 520, 0, 1, 0), (3553, 448, 1, 1, 0), (27779, 576, 1, 1, 0), (5861, 1024, 0, 1, 0), (16385, 1024, 1, 1, 1), (16257, 1032, 1, 1, 0), (72675, 704, 1, 0, 1), (16001, 1000, 0, 1, 1), (62501, 800, 0, 1, 1),
    (2931, 2048, 0, 1, 0), (8193, 2048, 1, 1, 1), (7783, 2056, 0, 1, 0), (16667, 3000, 1, 0, 1), (5571, 3592, 1, 0, 1), (4097, 4096, 0, 1, 1), (4097, 4096, 1, 1, 1),
    (445, 4096, 1, 1, 0), (297, 4104, 0, 0, 1), (1463, 4104, 0, 1, 1), (1220, 4104, 1, 1, 1), (297, 6144, 1, 0, 1), (977, 6144, 0, 1, 1),
    (2728, 6152, 1, 1, 0), (3252, 6152, 1, 0, 1), (1115, 7176, 0, 1, 1), (733, 8192, 0, 1, 0), (611, 8192, 1, 1, 0), (2049, 8192, 0, 1, 1)])
def test_rmsnorm_through_rings(T, H, with_res, forward, backward):
    from aws_ofi_nccl_b200.ops import _lib

    assert [_lib.load().b200_rmsnorm_ring(T, H, with_res, b) for b in (0, 1)] == [forward, backward]
    test_rmsnorm(T, H, bool(with_res))
    assert _lib.read_status() == 0


@pytest.mark.parametrize("T,F", [(1, 8), (3, 72), (257, 520), (1000, 2056), (4096, 1376)])
def test_swiglu(T, F):
    from aws_ofi_nccl_b200.ops import llm

    gu = (torch.randn(T, 2 * F, device="cuda") * 3).bfloat16()
    gu[0, :4] = torch.tensor([-100.0, 100.0, -88.0, 0.0], device="cuda")   # both ends of the exponential
    gu.requires_grad_(True)
    d = torch.randn(T, F, device="cuda").bfloat16()
    out = llm.swiglu(gu)
    (dgu,) = torch.autograd.grad(out, (gu,), d)
    g, u = gu.detach().double().split(F, -1)
    s = torch.sigmoid(g)
    _within(out.detach(), g * s * u, 2 * BF, 1e-35)
    D = d.double()
    _within(dgu, torch.cat((D * u * s * (1 + g * (1 - s)), D * g * s), -1), 2 * BF, 2.0 ** -20 * (D.abs() * u.abs()).max().item())


@pytest.mark.parametrize("hd,nq,nkv", [(64, 4, 2), (128, 3, 1), (20, 2, 1), (40, 2, 2)])
@pytest.mark.parametrize("layout", ["tokens", "heads"])
def test_rope_qkv(hd, nq, nkv, layout):
    from aws_ofi_nccl_b200.ops import llm

    B, S = 2, 37
    qkv = torch.randn(B * S, (nq + 2 * nkv) * hd, device="cuda").bfloat16().requires_grad_(True)
    ang = torch.rand(S + 3, hd // 2, device="cuda") * 6
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    outs = llm.rope_qkv(qkv, cos, sin, B, S, nq, nkv, hd)
    c, s = cos[:S].double().view(1, S, 1, -1), sin[:S].double().view(1, S, 1, -1)

    def turn(t, sign):
        a, b = t.double().split(hd // 2, -1)
        return torch.cat((a * c - sign * b * s, b * c + sign * a * s), -1)

    parts = qkv.detach().view(B, S, nq + 2 * nkv, hd).split((nq, nkv, nkv), 2)
    for got, part, rotated in zip(outs, parts, (True, True, False)):
        _within(got.detach(), turn(part, 1) if rotated else part.double(), BF, 2.0 ** -7)
    grads = [torch.randn_like(o) for o in outs]
    if layout == "heads":   # as attention returns them: a transposed [B, heads, S, hd]
        grads = [g.transpose(1, 2).contiguous().transpose(1, 2) for g in grads]
    (d,) = torch.autograd.grad(outs, (qkv,), grads)
    want = torch.cat((turn(grads[0], -1), turn(grads[1], -1), grads[2].double()), 2).view(B * S, -1)
    _within(d, want, BF, 2.0 ** -7)   # the two products of a rotation cancel: an error of one bf16 step of them


def test_nothing_is_differentiated_through_overwritten_logits():
    """Afterwards they hold the loss's gradient: what else is derived from them has no gradient of its own."""
    from aws_ofi_nccl_b200.ops import llm

    leaf = torch.randn(6, 64, device="cuda").bfloat16().requires_grad_(True)
    targets = torch.arange(6, device="cuda")
    logits = leaf * 1.0
    loss = llm.cross_entropy(logits, targets)
    with pytest.raises(RuntimeError, match="overwrites"):
        torch.autograd.grad(logits.float().sum(), leaf, retain_graph=True)
    with pytest.raises(RuntimeError, match="overwrites"):
        torch.autograd.grad(loss + logits.float().square().sum(), leaf, retain_graph=True)
    (d,) = torch.autograd.grad(loss, leaf)
    assert torch.equal(d, logits.detach())


@pytest.mark.parametrize("F", [8, 72])
def test_swiglu_of_rare_gates(F):
    """Infinities, NaN and gates at both ends of the range whose division is written out."""
    from aws_ofi_nccl_b200.ops import llm

    gate = torch.tensor([80.0, -80.0, 79.5, -79.5, 88.5, -88.0, 120.0, -120.0, math.inf, -math.inf, math.nan, 0.0, -0.0, 1e-38, 3e38, -3e38],
                        device="cuda")
    g = torch.zeros(gate.numel(), F, device="cuda")
    g[:, F // 2] = gate
    gu = torch.cat((g, torch.full_like(g, 0.75)), -1).bfloat16().requires_grad_(True)
    out = llm.swiglu(gu)
    d = torch.full_like(out, 0.5)
    (dgu,) = torch.autograd.grad(out, (gu,), d)
    gf = gu.detach()[:, :F].float()
    s = 1 / (1 + torch.exp(-gf))
    want = gf / (1 + torch.exp(-gf)) * 0.75
    silu = gf * s
    want_d = torch.cat((0.5 * 0.75 * (s + silu * (1 - s)), 0.5 * silu), -1)
    for a, b in ((out, want), (dgu, want_d)):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.bfloat16().isinf())
        ok = b.isfinite()
        _within(a.detach()[ok], b[ok].double(), 2 * BF, 1e-30)


def _misses(got, exact):
    """Elements that are not the exact value rounded to bf16. With a mean error of E ulp of 32 bits before that rounding a share of
    E / 2^16 is to be expected: as often lies the middle between two bf16 values in between."""
    return (got != exact.bfloat16()).sum().item() / got.numel() * 2.0 ** 16


def test_swiglu_errs_by_ulps_of_32_bits():
    """Its quotients and exponential are not correctly rounded; what is left of that in bf16 says by how much they err."""
    from aws_ofi_nccl_b200.ops import llm

    g = torch.Generator(device="cuda").manual_seed(5)
    gu = (torch.randn(2048, 2 * 4096, device="cuda", generator=g) * 3).bfloat16().requires_grad_(True)
    d = torch.randn(2048, 4096, device="cuda", generator=g).bfloat16()
    out = llm.swiglu(gu)
    (dgu,) = torch.autograd.grad(out, (gu,), d)
    G, U = gu.detach().double().split(4096, -1)
    s, D = torch.sigmoid(G), d.double()
    # two roundings and the exponential's error each; d(gate) has six, and terms that cancel
    assert _misses(out.detach(), G * s * U) < 2 and _misses(dgu[:, 4096:], D * G * s) < 2
    assert _misses(dgu[:, :4096], D * U * s * (1 + G * (1 - s))) < 8


@pytest.mark.parametrize("T,F", [(1, 32), (5, 96), (1000, 2080)])
def test_interleaved_swiglu_gradient_is_that_of_halves(T, F):
    """Gate and up alternate in blocks of 32 columns there: the same bits elsewhere."""
    from aws_ofi_nccl_b200.ops import _lib

    lib, d, gu = _lib.load(), torch.randn(T, F, device="cuda").bfloat16(), torch.randn(T, 2 * F, device="cuda").bfloat16()
    half, mixed = torch.empty_like(gu), torch.full_like(gu, 7.0)
    assert lib.b200_swiglu_bwd(d.data_ptr(), gu.data_ptr(), half.data_ptr(), T, F, _lib.stream_ptr()) == 0

    def interleave(t):
        return t.view(T, 2, F // 32, 32).transpose(1, 2).reshape(T, 2 * F).contiguous()

    inter = interleave(gu)
    assert lib.b200_swiglu_bwd_interleaved(d.data_ptr(), inter.data_ptr(), mixed.data_ptr(), T, F, _lib.stream_ptr()) == 0
    assert torch.equal(mixed, interleave(half))


@pytest.mark.parametrize("n", [8, 1024, 8 * 256 * 148 * 256 + 8])   # one vector; less than a CTA; one pass more than a full grid
def test_adamw_over_the_whole_grid(n):
    from aws_ofi_nccl_b200.ops import llm

    p, g = torch.randn(n, device="cuda").bfloat16(), torch.randn(n, device="cuda").bfloat16()
    m, v = torch.randn(n, device="cuda") * 0.1, torch.rand(n, device="cuda") * 0.01
    w = p.float()
    w0, terms = w.double(), 0.9 * m.double().abs() + 0.1 * g.double().abs()
    em, ev = 0.9 * m.double() + 0.1 * g.double(), 0.95 * v.double() + 0.05 * g.double() ** 2
    per_m = 1e-2 / (1 - 0.9 ** 3) / ((ev / (1 - 0.95 ** 3)).sqrt() + 1e-8)
    llm.adamw_step(p, g, m, v, w, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3)
    # fp32 holds 1 - beta to 4 ulp, 1 - beta^3 to 16; a handful of roundings besides
    ulp = 2.0 ** -24
    assert ((m - em).abs() <= 16 * ulp * terms).all() and ((v - ev).abs() <= 16 * ulp * ev).all()
    assert ((w - (w0 * (1 - 1e-2 * 0.1) - per_m * em)).abs() <= 4 * ulp * w0.abs() + 64 * ulp * per_m * terms).all()
    assert torch.equal(p, w.bfloat16()) and not g.any()

# a vector, a CTA's vectors and one more, more than the largest grid takes at once
@pytest.mark.parametrize("T,H", [(1, 8), (256, 8), (257, 8), (5, 4104), (9700, 8192)])
def test_embedding(T, H):
    from aws_ofi_nccl_b200.ops import llm

    g = torch.Generator(device="cuda").manual_seed(T + H)
    table, ids = torch.randn(50, H, device="cuda", generator=g).bfloat16(), torch.randint(0, 50, (T,), device="cuda", generator=g)
    assert torch.equal(llm.embedding(ids, table), table[ids])


LOWEST = torch.finfo(torch.bfloat16).min   # the usual value of a mask


# a vector, a thread's vectors (one to eight), a cluster of two to eight CTAs and the widest row that it holds, each with
# one element or vector more; the last is a row for two passes
@pytest.mark.parametrize("T,V", [(1, 1), (5, 7), (3, 2048), (300, 2049), (4, 4104), (7, 8200), (5, 16384), (40, 16392), (3, 32771),
                                 (6, 65544), (20, 128256), (2, 131072), (2, 131073)])
def test_cross_entropy(T, V):
    from aws_ofi_nccl_b200.ops import llm

    g = torch.Generator(device="cuda").manual_seed(T + V)
    pad = torch.full((T, (V + 7) // 8 * 8 + 8), 5.0, device="cuda").bfloat16()
    logits = pad[:, :V]
    logits.copy_(torch.randn(T, V, device="cuda", generator=g) * 3)
    if V > 64:
        logits[0, :48] = -math.inf   # whole vectors that are masked out
        logits[-1, V // 2:V // 2 + 3] = 60.0
    targets = torch.randint(0, V, (T,), device="cuda", generator=g)
    targets[0] = V - 1
    if T > 2:
        targets[1], targets[2] = -1, 0   # an ignored row
    x = logits.double()
    lse = torch.logsumexp(x, -1)
    counts = targets >= 0
    want_loss = torch.where(counts, lse - x.gather(1, targets.clamp_min(0)[:, None])[:, 0], torch.zeros_like(lse)).mean()
    want = torch.exp(x - lse[:, None])
    want.scatter_add_(1, targets.clamp_min(0)[:, None], -torch.ones_like(lse)[:, None])
    want = torch.where(counts[:, None], want / T, torch.zeros_like(want))
    loss = llm.cross_entropy(logits, targets)
    finite = lse.isfinite() & (x.gather(1, targets.clamp_min(0)[:, None])[:, 0].isfinite() | ~counts)
    assert finite.all()
    # exponentials of arguments up to 90 whose product with log2(e) is rounded to 24 bits, and sums of them
    err = 128 * 2.0 ** -24
    assert abs(loss.double() - want_loss) <= err * (1 + lse.abs().max())
    _within(logits, want, BF + err, err / T)
    assert (pad[:, V:] == 5).all()


# streamed rows: one chunk (24576 elements) and one vector more, all that the ring holds (98304) and one more, whole rings and more a second time; one
# row, several for a CTA, ragged widths; two rows for an SM in two passes
@pytest.mark.parametrize("T,V", [(1, 16392), (150, 16401), (700, 24576), (700, 24584), (200, 49153), (300, 32776), (160, 98304), (150, 98312), (2, 131080),
                                 (149, 196609), (2, 600007), (200, 24576)])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -10])   # small powers count, and do not
def test_cross_entropy_of_wide_rows(T, V, scale):
    from aws_ofi_nccl_b200.ops import _lib

    assert _lib.load().b200_cross_entropy_ctas(T, V) == 0
    g = torch.Generator(device="cuda").manual_seed(T + V)
    pad = torch.full((T, (V + 7) // 8 * 8 + 8), 5.0, device="cuda").bfloat16()
    logits = pad[:, :V]
    logits.copy_(torch.randn(T, V, device="cuda", generator=g) * 3)
    logits[0, :V // 2] = LOWEST
    logits[-1, V - 1] = 90.0   # the last element, alone in its sum: the others are small powers
    targets = torch.randint(0, V, (T,), device="cuda", generator=g)
    targets[0] = V - 1
    if T > 2:
        targets[1] = V
    counts = targets < V
    at = targets.clamp_max(V - 1)[:, None]
    rows = [0, T - 1] + ([1, T // 2] if T > 2 else [])
    x, loss = logits[rows].double(), torch.full((T,), math.nan, device="cuda")
    lse = torch.logsumexp(x, -1)
    want_loss = (lse - x.gather(1, at[rows])[:, 0]) * counts[rows]
    want = (x - lse[:, None]).exp()
    want.scatter_add_(1, at[rows], -torch.ones_like(lse)[:, None])
    want *= counts[rows][:, None] * scale
    rc = _lib.load().b200_cross_entropy(pad.data_ptr(), targets.data_ptr(), loss.data_ptr(), T, V, pad.stride(0), scale, _lib.stream_ptr())
    assert rc == 0 and (pad[:, V:] == 5).all() and loss.isfinite().all() and logits.isfinite().all() and (logits[counts] != 0).any(-1).all()
    # exponentials of arguments up to 110 whose product with log2(e) is rounded to 24 bits, and sums of them; a bf16 has no steps below 2^-133
    err = 160 * 2.0 ** -24
    _within(loss[rows], want_loss, err, err * (1 + lse.abs().max()))
    _within(logits[rows], want, BF + err, scale * err + 2.0 ** -133)
    assert _lib.read_status() == 0


# one chunk, two, all that the ring holds; one, two and four more that come a second time
@pytest.mark.parametrize("V", [16392, 32776, 98304, 98312, 131080, 180232])
def test_every_row_of_a_cta_of_the_streamed_cross_entropy(V):
    """Rows that follow one another through a CTA's ring: the slots that a row begins with change from row to row."""
    from aws_ofi_nccl_b200.ops import _lib

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    T = 5 * sms + 3   # six rows for CTAs 0 to 2, five for the others
    assert _lib.load().b200_cross_entropy_ctas(T, V) == 0
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.empty(T, V, device="cuda", dtype=torch.bfloat16).normal_(0, 3, generator=g)
    targets = torch.randint(0, V, (T,), device="cuda", generator=g)
    rows = torch.tensor([r for cta in (0, 2, 3, sms - 1) for r in range(cta, T, sms)], device="cuda")
    x, at = logits[rows].double(), targets[rows][:, None]
    lse = torch.logsumexp(x, -1)
    want_loss, want = lse - x.gather(1, at)[:, 0], (x - lse[:, None]).exp()
    want.scatter_add_(1, at, -torch.ones_like(lse)[:, None])
    loss = torch.full((T,), math.nan, device="cuda")
    assert _lib.load().b200_cross_entropy(logits.data_ptr(), targets.data_ptr(), loss.data_ptr(), T, V, V, 1.0, _lib.stream_ptr()) == 0
    # as above: arguments up to 40 whose product with log2(e) is rounded to 24 bits, and sums of their powers
    err = 160 * 2.0 ** -24
    _within(loss[rows], want_loss, err, err * (1 + lse.abs().max()))
    _within(logits[rows], want, BF + err, err + 2.0 ** -133)
    assert _lib.read_status() == 0


def test_rows_without_elements():
    """No loss, and no norm: what the entry points did before rows came through rings."""
    from aws_ofi_nccl_b200.ops import _lib

    lib, st = _lib.load(), _lib.stream_ptr()
    loss, targets = torch.full((3,), 7.0, device="cuda"), torch.zeros(3, device="cuda", dtype=torch.int64)
    buf = torch.zeros(64, device="cuda")
    assert lib.b200_cross_entropy(buf.data_ptr(), targets.data_ptr(), loss.data_ptr(), 3, 0, 0, 1.0, st) == 0
    assert (loss == 0).all()
    p = buf.data_ptr()
    rstd = torch.zeros(10000, device="cuda")
    assert lib.b200_rmsnorm_fwd(p, None, None, p, p, rstd.data_ptr(), 10000, 0, 1e-5, st) == 0
    torch.cuda.synchronize()
    assert _lib.read_status() == 0


def test_cross_entropy_of_a_row_with_nan_is_nan():
    from aws_ofi_nccl_b200.ops import llm

    logits = torch.randn(2, 128256, device="cuda").bfloat16()
    logits[0, 16384:32768] = math.nan   # all that one CTA holds
    targets = torch.zeros(2, device="cuda", dtype=torch.int64)
    assert llm.cross_entropy(logits, targets).isnan()


def _loss_and_gradient(rows, targets):
    """Loss of every row and gradient (scaled by 1) of rows that lie in a wider buffer, which stays as it is."""
    from aws_ofi_nccl_b200.ops import _lib

    T, V = rows.shape
    pad = torch.full((T, (V + 7) // 8 * 8 + 8), 5.0, device="cuda").bfloat16()
    pad[:, :V] = rows
    loss = torch.full((T,), math.nan, device="cuda")
    rc = _lib.load().b200_cross_entropy(pad.data_ptr(), targets.data_ptr(), loss.data_ptr(), T, V, pad.stride(0), 1.0, _lib.stream_ptr())
    assert rc == 0 and (pad[:, V:] == 5).all()
    return loss, pad[:, :V]


# rows of one CTA, of a cluster of two, four and eight, too many of them (two passes), and a wider row than a cluster holds
CE_PATHS = [(6, 2045), (6, 24587), (6, 40003), (6, 131069), (700, 24587), (6, 131075)]


@pytest.mark.parametrize("T,V", CE_PATHS)
@pytest.mark.parametrize("fill", [LOWEST, -math.inf, math.inf, math.nan, 3e38])
def test_cross_entropy_of_an_ignored_row_is_zero(T, V, fill):
    """Loss and gradient, whatever its logits hold."""
    rows = torch.randn(T, V, device="cuda").bfloat16()
    rows[::2] = fill
    targets = torch.full((T,), 3, device="cuda")
    targets[::2] = -1
    targets[2] = V
    loss, grad = _loss_and_gradient(rows, targets)
    assert (loss[::2] == 0).all() and (grad[::2] == 0).all()
    assert loss[1::2].isfinite().all() and (grad[1::2] != 0).any(-1).all()


@pytest.mark.parametrize("T,V", CE_PATHS)
def test_cross_entropy_at_both_ends_of_the_range(T, V):
    """Masks of the lowest value, as a whole row, as all that some CTAs of a cluster hold and beside a huge maximum; equal logits far
    from zero, whose distribution is uniform; every path against 64 bits."""
    base = torch.randn(6, V, device="cuda").bfloat16()
    targets = torch.tensor([3, V - 1, 5, 5, 1, V // 2], device="cuda")
    base[0] = LOWEST
    base[1, :V // 2] = LOWEST
    base[2, 5:8] = 3e38
    base[3], base[3, 5], base[3, 9] = LOWEST, -3e38, -3e38
    base[4], base[5] = 5013504.0, -999424.0
    rows, targets = base.repeat(T // 6 + 1, 1)[:T], targets.repeat(T // 6 + 1)[:T]
    x = rows.double()
    m = x.amax(-1, keepdim=True)
    lse = (x - m).exp().sum(-1).log()   # less the maximum
    want = (x - m - lse[:, None]).exp()
    want.scatter_add_(1, targets[:, None], -torch.ones_like(m))
    loss, grad = _loss_and_gradient(rows, targets)
    err = 64 * 2.0 ** -24   # exponentials of arguments down to -20 whose product with log2(e) is rounded, and sums of them
    _within(loss, lse + (m - x.gather(1, targets[:, None]))[:, 0], err, err)
    _within(grad, want, BF + err, 1e-38)


@pytest.mark.parametrize("T,K", [(1, 8), (9, 256), (17, 264), (5, 512), (9, 520), (3, 1032), (7, 2056), (300, 4096), (5, 4104), (3, 8200),
                                 (2, 16384), (3, 16392), (1200, 16400)])
def test_quantize_rows_fp8(T, K):
    """Bit for bit: the scale is amax / 448, the values are rounded once."""
    from aws_ofi_nccl_b200.ops.gemm import quantize_rows_fp8

    x = torch.randn(T, K + 8, device="cuda").bfloat16()[:, :K]
    x[0] *= 1e-3
    if T > 2:
        x[2] = 0
    q, s = quantize_rows_fp8(x)
    scale = x.float().abs().amax(-1).clamp_min(1e-12) * (1.0 / 448.0)
    assert torch.equal(s, scale)
    want = (x.float() * (1.0 / scale)[:, None]).clamp(-448, 448).to(torch.float8_e4m3fn)
    assert torch.equal(q.view(torch.uint8), want.view(torch.uint8))
