"""MoE dispatch and combine on one rank, where every row stays local: the received rows, the raw
collectives' window contents and the gradients, against sums in 64 bits."""
import pytest
import torch
import torch.distributed as dist

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


# a team of one warp, of several, of the whole CTA with one column step; then rows of several steps (ragged, full,
# the largest), several tokens per team, several teams of one warp with a ragged last group
@pytest.mark.parametrize("T,H,E,k", [(1, 256, 8, 1), (37, 512, 16, 3), (130, 1280, 64, 5), (64, 2048, 8, 8),
                                     (37, 2304, 16, 3), (21, 7168, 64, 8), (9, 8192, 8, 2), (2500, 1280, 16, 2), (1300, 4096, 8, 1),
                                     (10003, 256, 8, 1)])
@pytest.mark.parametrize("fp8", [False, True])
def test_roundtrip_and_gradients(comm, T, H, E, k, fp8):
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    ep = ExpertParallel(comm, T, H, E, k)
    g = torch.Generator(device="cuda").manual_seed(T + H + E)
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16().requires_grad_(True)
    dy = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    w, idx = torch.topk(torch.softmax(torch.randn(T, E, device="cuda", generator=g), -1), k, dim=-1)
    idx = idx.to(torch.int32).contiguous()
    if T > 1:
        idx[-1, 0] = -1   # a slot that goes nowhere
    w = w.contiguous().requires_grad_(True)
    sent = (idx >= 0).double()
    rows = ep.dispatch(x, idx, w, fp8)
    n = int(ep.expert_offsets[-1].item())
    assert n == int(sent.sum().item())
    meta = ep.recv_meta()[:n].cpu()
    src = x.detach()[meta[:, 0].long()]
    step = 2.0 ** -4 if fp8 else 0.0   # e4m3 keeps four significant bits
    got = rows.detach()
    assert ((got[:n].float() - src.float()).abs() <= step * src.float().abs() + (1e-2 if fp8 else 0)).all()
    assert (got[n:] == 0).all()
    out = ep.combine(rows, w)
    per_slot = torch.zeros(T, k, H, device="cuda", dtype=torch.float64)
    per_slot[meta[:, 0].long(), meta[:, 1].long()] = got[:n].double()
    W = w.detach().double()
    BF = 2.0 ** -8
    mag = (W[..., None] * per_slot).abs().sum(1)
    want = (W[..., None] * per_slot).sum(1)
    assert ((out.detach().double() - want).abs() <= BF * want.abs() + 1e-6 * mag + 1e-6).all()
    dx, dw = torch.autograd.grad(out, (x, w), dy)
    D = dy.double()
    total = (W * sent).sum(1, keepdim=True)
    assert ((dx.double() - D * total).abs() <= 2 * BF * (D * total).abs() + 1e-6).all()   # w * dy is rounded, then their sum
    want_w = (D[:, None] * per_slot).sum(-1) * sent
    assert ((dw.double() - want_w).abs() <= 1e-5 * (D[:, None] * per_slot).abs().sum(-1) + 1e-6).all()


def test_raw_calls_leave_rows_and_cells_in_the_window(comm):
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    T, H, E, k = 50, 512, 8, 2
    ep = ExpertParallel(comm, T, H, E, k)
    x = torch.randn(T, H, device="cuda").bfloat16()
    idx = torch.randint(0, E, (T, k), device="cuda", dtype=torch.int32)
    ep.route(idx)
    ep.dispatch_raw(x, idx, None, fp8=False)
    meta = ep.recv_meta()[: T * k]
    assert torch.equal(ep.recv_rows(False)[: T * k], x[meta[:, 0].long()])
    out = torch.empty_like(x)
    ep.combine_raw(ep.recv_rows(False)[: T * k].clone(), None, out)
    assert torch.equal(ep.combine_cells(), x[:, None].expand(T, k, H))
    assert torch.equal(out, (2 * x.float()).bfloat16())


@pytest.mark.parametrize("T,H,E,k", [(1, 256, 8, 1), (50, 512, 8, 2), (70, 2304, 16, 3)])
def test_views_of_the_window_hold_what_the_differentiable_calls_moved(comm, T, H, E, k):
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    ep = ExpertParallel(comm, T, H, E, k)
    g = torch.Generator(device="cuda").manual_seed(T + H)
    x, dy = (torch.randn(T, H, device="cuda", generator=g).bfloat16() for _ in range(2))
    x.requires_grad_(True)
    w, idx = torch.topk(torch.softmax(torch.randn(T, E, device="cuda", generator=g), -1), k, dim=-1)
    idx, w = idx.to(torch.int32).contiguous(), w.contiguous().requires_grad_(True)
    ep.recv_rows(False).fill_(7.0)
    ep.combine_cells().fill_(7.0)
    rows = ep.dispatch(x, idx, w)
    meta = ep.recv_meta()[: T * k].long()
    token, slot = meta[:, 0], meta[:, 1]
    assert torch.equal(ep.recv_rows(False)[: T * k], x.detach()[token])
    assert torch.equal(rows.detach()[: T * k], x.detach()[token])
    out = ep.combine(rows, w)
    assert torch.equal(ep.combine_cells(), x.detach()[:, None].expand(T, k, H))
    out.backward(dy)
    # the backward pass sends w * dy along the same rows and gathers what came back into the same cells
    sent = (w.detach()[token, slot][:, None] * dy[token].float()).bfloat16()
    assert torch.equal(ep.recv_rows(False)[: T * k], sent)
    assert torch.equal(ep.combine_cells()[token, slot], sent)


def test_an_earlier_routing_is_continued_from_its_saved_rows(comm):
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    T, H, E, k = 60, 256, 16, 2
    ep = ExpertParallel(comm, T, H, E, k)
    g = torch.Generator(device="cuda").manual_seed(5)
    batches = []
    for _ in range(2):
        x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
        idx = torch.rand(T, E, device="cuda", generator=g).topk(k, dim=-1).indices.to(torch.int32).contiguous()
        ep.route(idx)
        ep.dispatch_raw(x, idx, None, fp8=False)
        batches.append((x, idx, ep.row_of.clone(), ep.expert_offsets.clone()))
    x, idx, row_of, offsets = batches[0]
    ep.row_of.copy_(row_of)
    ep.expert_offsets.copy_(offsets)
    ep.dispatch_raw(x, idx, None, fp8=False, use_saved_rows=True)
    out = torch.empty_like(x)
    ep.combine_raw(ep.recv_rows(False)[: T * k].clone(), None, out)
    assert torch.equal(out, (2 * x.float()).bfloat16())


def test_collect_copies_what_other_ranks_sent(comm):
    """Records name another rank for half of the rows, as after a dispatch of two ranks."""
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    T, H, E, k = 700, 768, 8, 2
    ep = ExpertParallel(comm, T, H, E, k, capacity_factor=1.5)
    idx = torch.randint(0, E, (T, k), device="cuda", dtype=torch.int32)
    idx[5:30, 0] = -1   # fewer rows than capacity
    ep.route(idx)
    ep.dispatch_raw(torch.randn(T, H, device="cuda").bfloat16(), idx, None, fp8=False)
    n = int(ep.expert_offsets[-1].item())
    assert n == T * k - 25 < ep.capacity
    remote = torch.rand(n, device="cuda") < 0.5
    ep.recv_meta()[:n, 3] = remote.int()
    window = ep.recv_rows(False)[:n].clone()
    own = torch.full((ep.capacity, H), 3.0, device="cuda", dtype=torch.bfloat16)
    got = ep.collect(own.clone(), True)
    assert torch.equal(got[:n], torch.where(remote[:, None], window, own[:n])) and (got[n:] == 0).all()
    got = ep.collect(own.clone(), False)
    assert torch.equal(got[:n], window) and (got[n:] == 0).all()


@pytest.mark.parametrize("T,H,k", [(40, 256, 2), (600, 768, 5), (21, 7168, 8)])
def test_combine_sums_own_rows_and_delivered_cells(comm, T, H, k):
    """Half of the cells are planted in the window, as another rank delivers them; the others come from y."""
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    E = 16
    ep = ExpertParallel(comm, T, H, E, k)
    g = torch.Generator(device="cuda").manual_seed(T)
    idx = torch.rand(T, E, device="cuda", generator=g).topk(k, dim=-1).indices.to(torch.int32).contiguous()
    ep.route(idx)
    ep.dispatch_raw(torch.randn(T, H, device="cuda", generator=g).bfloat16(), idx, None, fp8=False)
    y = torch.randn(T * k, H, device="cuda", generator=g).bfloat16()
    w = torch.rand(T, k, device="cuda", generator=g)
    remote = torch.rand(T, k, device="cuda", generator=g) < 0.5
    delivered = torch.randn(T, k, H, device="cuda", generator=g).bfloat16()
    cells = torch.where(remote[..., None], delivered, y[ep.row_of.long()])
    ep.combine_cells().copy_(torch.where(remote[..., None], delivered, torch.full_like(delivered, 9.0)))
    ep.local_row[remote] = -1
    out, kept = torch.empty(T, H, device="cuda", dtype=torch.bfloat16), torch.empty_like(cells)
    ep.combine_raw(y, w, out, cells_out=kept)
    assert torch.equal(kept, cells) and torch.equal(ep.combine_cells(), cells)
    terms = w.double()[..., None] * cells.double()
    # fp32 sums of k products, one rounding to bf16
    assert ((out.double() - terms.sum(1)).abs() <= 2.0 ** -8 * terms.sum(1).abs() + (k + 1) * 2.0 ** -24 * terms.abs().sum(1)).all()


@pytest.mark.parametrize("T,H,k", [(1, 256, 1), (40, 1280, 3), (700, 768, 2), (3000, 768, 4)])
def test_fp8_rows_are_those_of_the_window(comm, T, H, k):
    """Dispatch stores this rank's rows as the values that their fp8 payload stands for; rows whose records name another
    rank come from the window, rows that nobody sent are zeros."""
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    E = 8
    ep = ExpertParallel(comm, T, H, E, k, capacity_factor=1.5)
    g = torch.Generator(device="cuda").manual_seed(T + H)
    idx = torch.rand(T, E, device="cuda", generator=g).topk(k, dim=-1).indices.to(torch.int32).contiguous()
    idx[T // 2:T // 2 + 30, 0] = -1   # fewer rows than capacity
    x, w = torch.randn(T, H, device="cuda", generator=g).bfloat16(), torch.rand(T, k, device="cuda", generator=g)
    rows = ep.dispatch(x, idx, w, True)
    assert torch.equal(rows, ep.dequant())
    n = int(ep.expert_offsets[-1].item())
    remote = torch.rand(n, device="cuda", generator=g) < 0.5
    ep.recv_meta()[:n, 3] = remote.int()
    own = torch.full_like(rows, 3.0)
    got = ep.collect_fp8(own.clone())
    assert torch.equal(got[:n], torch.where(remote[:, None], rows[:n], own[:n])) and (got[n:] == 0).all()
    # weighted rows are scaled and quantised one by one
    ep.dispatch_raw(x, idx, w, fp8=True, use_saved_rows=True, scale_by_weight=True, local_out=own)
    assert torch.equal(own[:n], ep.dequant()[:n])


# one expert, an odd number, one per thread and one more, several per thread, as many as there may be; ragged and few tokens
@pytest.mark.parametrize("E", [1, 3, 256, 257, 700, 1024])
@pytest.mark.parametrize("T", [1, 1001])
def test_route_counts_the_rows_of_every_expert(comm, E, T):
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    ep = ExpertParallel(comm, T, 256, E, 3)
    for seed in range(2):
        g = torch.Generator(device="cuda").manual_seed(E + T + seed)
        idx = torch.randint(-1, E, (T, 3), device="cuda", generator=g, dtype=torch.int32)   # -1 goes nowhere
        offsets = ep.route(idx)
        counts = torch.bincount(idx[idx >= 0].long(), minlength=E)
        assert offsets[0] == 0 and torch.equal(offsets[1:].long(), counts.cumsum(0))
        assert torch.equal(ep.dest_base.long(), counts.cumsum(0) - counts)


# more tokens than CTAs of dispatch, sum and weight gradient at once work on, call after call
def test_more_tokens_than_a_grid_holds(comm):
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    T, H, E = 40001, 256, 8
    ep = ExpertParallel(comm, T, H, E, 1, capacity_factor=1.0)
    g = torch.Generator(device="cuda").manual_seed(5)
    for _ in range(3):
        x, dy = (torch.randn(T, H, device="cuda", generator=g).bfloat16() for _ in range(2))
        x.requires_grad_(True)
        idx = torch.randint(0, E, (T, 1), device="cuda", generator=g, dtype=torch.int32)
        w = torch.full((T, 1), 0.5, device="cuda", requires_grad=True)
        out = ep.combine(ep.dispatch(x, idx, w), w)
        assert torch.equal(out, x.detach() * 0.5)   # a power of two: nothing is rounded
        dx, dw = torch.autograd.grad(out, (x, w), dy)
        want = (dy.double() * x.detach().double()).sum(-1, keepdim=True)
        mag = (dy.double() * x.detach().double()).abs().sum(-1, keepdim=True)
        assert torch.equal(dx, dy * 0.5) and ((dw.double() - want).abs() <= H * 2.0 ** -24 * mag).all()


# fewer tokens than an SM's CTAs take, more than one grid holds
@pytest.mark.parametrize("T", [50, 9001])
@pytest.mark.parametrize("fp8", [False, True])
def test_dispatch_and_combine_between_products(comm, T, fp8):
    """Kernels that come up while the one before ends: products that make the rows, take them and give them back, pass after pass without a wait,
    give the same bits as with one after every call."""
    from aws_ofi_nccl_b200.ops.gemm import gemm
    from aws_ofi_nccl_b200.parallel.expert_parallel import ExpertParallel

    H, E = 256, 8
    ep = ExpertParallel(comm, T, H, E, 1, capacity_factor=1.0)
    g = torch.Generator(device="cuda").manual_seed(T)
    x0 = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    w1, w2 = ((torch.randn(H, H, device="cuda", generator=g) * H ** -0.5).bfloat16() for _ in range(2))
    idx = torch.randint(0, E, (T, 1), device="cuda", generator=g, dtype=torch.int32)
    weights = torch.rand(T, 1, device="cuda", generator=g)

    def passes(wait):
        x, outs = x0.clone(), []

        def done():
            if wait:
                torch.cuda.synchronize()

        for _ in range(3):
            sent = gemm(x, w1)
            done()
            rows = ep.dispatch(sent, idx, weights, fp8)
            done()
            made = gemm(rows, w2)
            done()
            back = ep.combine(made, weights)
            done()
            x = gemm(back, w1)
            done()
            outs += [sent, back, x]
        return outs

    with torch.no_grad():
        want, got = passes(True), passes(False)
    for a, b in zip(want, got):
        assert torch.equal(a, b)
