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


@pytest.mark.parametrize("T,H,E,k", [(1, 256, 8, 1), (37, 512, 16, 3), (130, 1280, 64, 5), (64, 2048, 8, 8)])
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
