"""The native layers (linear, RMSNorm, SwiGLU, rotary split) as callables: what they refuse, and that
they can be traced."""
import ctypes

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


def test_layers_refuse_what_their_kernels_cannot_read():
    from aws_ofi_nccl_b200.ops import llm

    def bf(*shape):
        return torch.zeros(*shape, dtype=torch.bfloat16)

    for call in (lambda: llm.rmsnorm(bf(4, 16), bf(16)),                      # not on a GPU
                 lambda: llm.rmsnorm(torch.zeros(4, 16), torch.zeros(16)),    # not bfloat16
                 lambda: llm.swiglu(bf(4, 16)),
                 lambda: llm.swiglu(torch.zeros(4, 16))):
        with pytest.raises(AssertionError):
            call()


@pytest.mark.parametrize("name,args", [
    ("b200_rmsnorm_fwd", lambda p: (p[0], p[1], p[2], p[3], p[4], 64, 4, 64, 1e-5, None)),
    ("b200_rmsnorm_bwd", lambda p: (p[0], p[1], p[2], 64, p[3], p[4], p[5], 64, 0, 4, 64, None)),
    ("b200_swiglu_fwd", lambda p: (p[0], p[1], 4, 64, None)),
    ("b200_swiglu_bwd", lambda p: (p[0], p[1], p[2], 4, 64, None)),
    ("b200_swiglu_bwd_interleaved", lambda p: (p[0], p[1], p[2], 4, 64, None)),
])
def test_entry_points_refuse_a_misaligned_pointer(name, args):
    """Refused before anything is launched: the addresses are made up."""
    from aws_ofi_nccl_b200.ops import _lib

    if torch.cuda.is_available():
        pytest.skip("made-up addresses stay off the GPU")
    fn = getattr(_lib.load(), name)
    used = []
    args(type("P", (), {"__getitem__": lambda self, i: used.append(i)})())
    for bad in set(used):
        ptrs = [4096 * (i + 1) + (2 if i == bad else 0) for i in range(8)]
        assert fn(*args(ptrs)) == 10001


@pytest.mark.parametrize("name,args", [
    ("b200_embedding_fwd", lambda p: (4096, p, 8192, 4, 64, None)),
    ("b200_embedding_fwd", lambda p: (4096, 8192, p, 4, 64, None)),
    ("b200_embedding_bwd", lambda p: (4096, p, 8192, 4, 64, None)),
    ("b200_embedding_bwd", lambda p: (4096, 8192, p, 4, 64, None)),
])
def test_the_embedding_refuses_a_misaligned_pointer(name, args):
    """As above, refused before anything is launched: the addresses are made up."""
    from aws_ofi_nccl_b200.ops import _lib

    if torch.cuda.is_available():
        pytest.skip("made-up addresses stay off the GPU")
    assert getattr(_lib.load(), name)(*args(16386)) == 10001


@pytest.mark.parametrize("V", [8, 1000, 16392, 131080])
def test_the_cross_entropy_refuses_misaligned_logits(V):
    """On every path, before anything is launched."""
    from aws_ofi_nccl_b200.ops import _lib

    if torch.cuda.is_available():
        pytest.skip("made-up addresses stay off the GPU")
    assert _lib.load().b200_cross_entropy(16386, 4096, 8192, 4, V, (V + 7) // 8 * 8, 1.0, None) == 10001


@pytest.mark.parametrize("T,V,ctas", [
    (1, 8, 1), (100000, 16384, 1), (1, 131073, 0), (0, 8, 0),
    (1, 24576, 2), (74, 24576, 2), (92, 24576, 0), (200, 32768, 2), (296, 32768, 0), (4, 40000, 4), (55, 40000, 4), (111, 40000, 0), (111, 65536, 4),
    (148, 65536, 0), (37, 65544, 8), (74, 131072, 8), (1, 16392, 0), (148, 16392, 0), (148, 50264, 0), (148, 65544, 0), (92, 73000, 0)])
def test_rows_of_the_cross_entropy_take_the_faster_way(T, V, ctas):
    """CTAs that share a row as measured on 148 SMs, 0 for two passes."""
    from aws_ofi_nccl_b200.ops import _lib

    assert _lib.load().b200_cross_entropy_ctas(T, V) == ctas


@pytest.mark.parametrize("T,H,with_res,backward,ring", [
    (65536, 64, 0, 0, 0), (65536, 64, 0, 1, 0), (262144, 192, 1, 0, 0), (8192, 128, 0, 0, 0), (65536, 256, 0, 0, 1), (20000, 256, 0, 0, 0), (65536, 256, 0, 1, 0),
    (1500, 2048, 0, 0, 0), (8192, 2048, 0, 0, 1), (3000, 3072, 0, 0, 0), (8192, 3072, 0, 0, 1), (4096, 4096, 1, 0, 1), (16384, 4096, 1, 0, 0), (16384, 4096, 0, 0, 1),
    (4096, 640, 1, 0, 0), (65536, 520, 1, 0, 1), (900, 3072, 1, 0, 0), (1500, 5120, 1, 0, 1), (600, 8192, 1, 0, 0),
    (4096, 2048, 0, 1, 0), (16384, 2048, 0, 1, 1), (16384, 2056, 0, 1, 0), (4096, 4096, 1, 1, 1), (4096, 5120, 0, 1, 1), (296, 4104, 0, 1, 0), (297, 4104, 0, 1, 1),
    (1500, 6152, 0, 1, 0), (4096, 8192, 0, 1, 1), (4096, 8192, 1, 1, 0), (0, 4096, 0, 0, 0), (1000000, 0, 0, 0, 0), (1000000, 0, 0, 1, 0)])
def test_rows_of_a_norm_take_the_faster_way(T, H, with_res, backward, ring):
    """Whether they come through a ring, as measured on 148 SMs on both sides of where that changes."""
    from aws_ofi_nccl_b200.ops import _lib

    assert _lib.load().b200_rmsnorm_ring(T, H, with_res, backward) == ring


def test_the_embedding_refuses_what_its_kernel_cannot_read():
    """Nothing here is on a GPU; what lies on one is tested below."""
    from aws_ofi_nccl_b200.ops import llm

    ids, table = torch.zeros(4, dtype=torch.int64), torch.zeros(3, 8, dtype=torch.bfloat16)
    with pytest.raises(AssertionError, match="ids"):
        llm.embedding(ids, table)


@pytest.mark.gpu
def test_the_embedding_refuses_other_types_and_layouts():
    from aws_ofi_nccl_b200.ops import llm

    ids, table = torch.arange(4, device="cuda"), torch.randn(6, 16, device="cuda").bfloat16()
    for bad, what in ((ids.int(), "ids"), (ids.cpu(), "ids"), (torch.arange(8, device="cuda")[::2], "ids")):
        with pytest.raises(AssertionError, match=what):
            llm.embedding(bad, table)
    for bad in (table.float(), table.cpu(), torch.randn(6, 24, device="cuda").bfloat16()[:, :16], table[0], table.T):
        with pytest.raises(AssertionError, match="table"):
            llm.embedding(ids, bad)
    assert torch.equal(llm.embedding(ids.cpu().pin_memory(), table), table[:4])   # read in place
    for buffer in (torch.zeros(6, 16, device="cuda"), torch.zeros(5, 16, device="cuda").bfloat16(), torch.zeros(6, 24, device="cuda").bfloat16()[:, :16]):
        leaf = table.clone().requires_grad_(True)
        leaf.main_grad = buffer
        with pytest.raises(AssertionError, match="gradient buffer"):
            llm.embedding(ids, leaf).sum().backward()
        assert not buffer.any()


@pytest.mark.gpu
def test_gradients_of_any_view_are_taken():
    """Contiguous gradients that start at an odd element, and a batch of one whose stride is odd."""
    from aws_ofi_nccl_b200.ops import llm

    def odd(*shape):
        n = torch.Size(shape).numel()
        return torch.randn(n + 1, device="cuda").bfloat16()[1:].view(*shape)

    x, r, w = (torch.randn(*s, device="cuda").bfloat16().requires_grad_(True) for s in ((5, 64), (5, 64), (64,)))
    gu = torch.randn(5, 64, device="cuda").bfloat16().requires_grad_(True)
    qkv = torch.randn(8, 128, device="cuda").bfloat16().requires_grad_(True)
    ang = torch.rand(8, 16, device="cuda")
    cases = [(lambda: llm.rmsnorm(x, w, residual=r), (x, r, w), [odd(5, 64), odd(5, 64)]),
             (lambda: (llm.swiglu(gu),), (gu,), [odd(5, 32)]),
             (lambda: llm.rope_qkv(qkv, ang.cos(), ang.sin(), 1, 8, 2, 1, 32), (qkv,),
              [odd(1, 8, 2, 32), odd(1, 8, 1, 32), torch.randn(300, device="cuda").bfloat16().as_strided((1, 8, 1, 32), (257, 32, 32, 1))])]
    for fn, inputs, grads in cases:
        got = torch.autograd.grad(fn(), inputs, grads)
        want = torch.autograd.grad(fn(), inputs, [g.clone(memory_format=torch.contiguous_format) for g in grads])
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
def test_layers_refuse_misaligned_and_misshapen_inputs():
    from aws_ofi_nccl_b200.ops import _lib, llm

    def odd(*shape):
        n = torch.Size(shape).numel()
        return torch.zeros(n + 1, device="cuda", dtype=torch.bfloat16)[1:].view(*shape)

    x, w = (torch.zeros(*s, device="cuda", dtype=torch.bfloat16) for s in ((5, 64), (64,)))
    for call in (lambda: llm.rmsnorm(odd(5, 64), w), lambda: llm.rmsnorm(x, odd(64)), lambda: llm.swiglu(odd(5, 64))):
        with pytest.raises(_lib.B200OpsError):
            call()
    for call in (lambda: llm.rmsnorm(x, w[:56]), lambda: llm.rmsnorm(x, w.float()), lambda: llm.rmsnorm(x, w, residual=x[:4]),
                 lambda: llm.swiglu(torch.zeros(16, 17, device="cuda", dtype=torch.bfloat16))):
        with pytest.raises(AssertionError):
            call()


def test_the_rotary_split_refuses_misaligned_tables():
    from aws_ofi_nccl_b200.ops import _lib

    if torch.cuda.is_available():
        pytest.skip("made-up addresses stay off the GPU")
    lib = _lib.load()
    strides = (ctypes.c_longlong * 9)(64, 32, 32, 64, 32, 32, 64, 32, 32)
    for cos, sin in ((4096 + 4, 8192), (4096, 8192 + 4)):
        args = [ctypes.c_void_p(64), ctypes.c_longlong(128), *(ctypes.c_void_p(64 * i) for i in (2, 3, 4)), strides,
                ctypes.c_void_p(cos), ctypes.c_void_p(sin), ctypes.c_longlong(2)]
        assert lib.b200_rope_qkv(*args, 1, 1, 32, 2, 0, None) == 10001
        assert lib.b200_rope(64, cos, sin, 2, 1, 32, 32, 2, 0, None) == 10001


@pytest.mark.gpu
@pytest.mark.parametrize("backward", [False, True])
def test_other_threads_run_while_a_launch_waits(backward):
    """A launch into a full queue waits for the GPU; the interpreter must not wait with it."""
    import threading
    import time

    from aws_ofi_nccl_b200.ops import gemm

    x = torch.randn(8, 64, device="cuda").bfloat16()
    w = torch.randn(64, 64, device="cuda").bfloat16()
    w.main_grad = torch.zeros_like(w)
    if backward:
        w.requires_grad_(True)
    scratch = torch.zeros(8, device="cuda").add_(1)   # every kernel is loaded before the queue is filled
    y = gemm.linear(x, w)
    if backward:
        y.backward(torch.randn_like(y))
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    outs = [gemm.linear(x, w) for _ in range(200)] if backward else None
    dy = torch.randn_like(outs[0]) if backward else None
    torch.cuda.synchronize()
    pause = 1_000_000_000   # clocks: about half a second
    torch.cuda._sleep(pause)
    depth, waited = 0, 0.0
    while waited < 0.05 and depth < 20000:    # launches until one waits
        t0 = time.perf_counter()
        scratch.add_(1)
        depth, waited = depth + 1, time.perf_counter() - t0
    torch.cuda.synchronize()
    thread = threading.Thread(target=tick)
    thread.start()
    torch.cuda._sleep(pause)
    for _ in range(depth - 20):
        scratch.add_(1)
    t0 = time.perf_counter()
    if backward:
        torch.autograd.backward(outs, [dy] * len(outs))   # one weight-gradient product each
    else:
        for _ in range(200):
            gemm.linear(x, w)
    issued = time.perf_counter() - t0
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    if issued < 0.2:
        pytest.skip("no launch waited for the queue")
    assert max(gaps) < issued / 2, (issued, max(gaps))


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["grad_written", "grad_ready"])
def test_an_exception_of_a_parameters_attribute_reaches_the_caller(where):
    from aws_ofi_nccl_b200.ops import gemm

    class Odd(Exception):
        pass

    class Raises:
        def __bool__(self):
            raise Odd

        def __call__(self, weight):
            raise Odd

    w = torch.randn(16, 16, device="cuda").bfloat16().requires_grad_(True)
    w.main_grad = torch.zeros_like(w)
    setattr(w, where, Raises())
    with pytest.raises(Odd):
        gemm.linear(torch.randn(8, 16, device="cuda").bfloat16(), w).float().sum().backward()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1,), (2, 65), (0, 4)])
def test_the_embedding_adds_its_gradient_up_from_any_view(shape):
    from aws_ofi_nccl_b200.ops import llm

    table = torch.randn(33, 72, device="cuda").bfloat16().requires_grad_(True)
    ids = torch.randint(0, 33, shape, device="cuda")
    d = torch.randint(-2, 3, (ids.numel() * 72 + 1,), device="cuda").bfloat16()[1:].view(*shape, 72)   # at an odd element; sums exact
    want = torch.zeros(33, 72, device="cuda").index_add_(0, ids.reshape(-1), d.reshape(-1, 72).float())
    for written in (None, False, True):   # an ordinary gradient, the first into the flat buffer, one added to it
        table.grad = None
        if written is not None:
            table.main_grad, table.grad_written = torch.ones(33, 72, device="cuda").bfloat16(), written
        out = llm.embedding(ids, table)
        assert torch.equal(out, table.detach()[ids])
        out.backward(d)
        got = table.grad if written is None else table.main_grad
        assert torch.equal(got.float(), want + (1 if written else 0))
    traced = torch.jit.trace(llm.embedding, (torch.zeros_like(ids), torch.zeros_like(table)), check_trace=False)
    assert torch.equal(traced(ids, table), out)


@pytest.mark.gpu
def test_the_cross_entropy_is_the_same_inside_and_outside_of_python():
    """Loss, gradient, what the logits hold, and what is refused."""
    from aws_ofi_nccl_b200.ops import llm

    g = torch.Generator(device="cuda").manual_seed(2)
    leaf = torch.randn(40, 96, device="cuda", generator=g).bfloat16().requires_grad_(True)
    targets = torch.randint(0, 96, (40,), device="cuda", generator=g)
    results = []
    for fn in (llm.cross_entropy, lambda *a: llm._CrossEntropy.apply(*a)[0]):
        logits = leaf[:, :72] * 1.0   # any row pitch
        version = logits._version
        loss = fn(logits, targets % 72)
        assert logits._version > version and loss.requires_grad and loss.shape == ()
        (d,) = torch.autograd.grad(loss * 3, leaf)   # the incoming scalar is taken for one
        with torch.no_grad():
            plain = fn(leaf.detach().clone(), targets)
        assert not plain.requires_grad
        results.append((loss.detach(), d, logits.detach(), plain))
        with pytest.raises(ValueError):
            fn(torch.zeros(8, device="cuda", dtype=torch.bfloat16), targets)
        with pytest.raises(AssertionError):
            fn(torch.zeros(96, 40, device="cuda", dtype=torch.bfloat16).T, targets)
        with pytest.raises(ZeroDivisionError):
            fn(torch.zeros(0, 96, device="cuda", dtype=torch.bfloat16), targets[:0])
        with pytest.raises(RuntimeError, match="leaf"):
            fn(leaf.detach().clone().requires_grad_(True), targets)
    assert all(torch.equal(a, b) for a, b in zip(*results))


def _cross_entropies():
    from aws_ofi_nccl_b200.ops import llm

    return llm.cross_entropy, lambda *a: llm._CrossEntropy.apply(*a)[0]


def test_the_cross_entropy_refuses_what_its_kernel_cannot_read():
    """Nothing here is on a GPU; what lies on one is tested below."""
    targets = torch.zeros(4, dtype=torch.int64)
    for fn in _cross_entropies():
        for logits in (torch.zeros(4, 16, dtype=torch.bfloat16), torch.zeros(4, 16)):
            with pytest.raises(AssertionError):
                fn(logits, targets)


@pytest.mark.gpu
def test_the_cross_entropy_refuses_other_types_and_targets():
    """Before anything is launched: the logits stay as they are."""
    logits, targets = torch.ones(8, 16, device="cuda").bfloat16(), torch.arange(8, device="cuda")
    for fn in _cross_entropies():
        for x, t in ((logits.float(), targets), (logits.half(), targets), (logits, targets.int()), (logits, targets.float()),
                     (logits, targets[:7]), (logits, torch.arange(16, device="cuda")[::2]), (logits, targets.cpu())):
            with pytest.raises(AssertionError):
                fn(x, t)
            assert (x == 1).all()
        for t in (targets.view(2, 4), torch.arange(9, device="cuda"), targets.cpu().pin_memory()):   # one for every row
            assert fn(logits.clone(), t).isfinite()


@pytest.mark.gpu
def test_the_cross_entropy_reads_its_switch_in_the_backward_pass(monkeypatch):
    """Cleared between the passes, the incoming scalar counts; set again before the backward pass, it does not."""
    from aws_ofi_nccl_b200.ops import llm

    g = torch.Generator(device="cuda").manual_seed(4)
    leaf = torch.randn(40, 96, device="cuda", generator=g).bfloat16().requires_grad_(True)
    targets = torch.randint(0, 96, (40,), device="cuda", generator=g)

    def gradient(before, between):
        monkeypatch.setattr(llm._CrossEntropy, "assume_unit_grad", before, raising=False)
        loss = llm.cross_entropy(leaf * 1.0, targets)
        monkeypatch.setattr(llm._CrossEntropy, "assume_unit_grad", between, raising=False)
        return torch.autograd.grad(loss * 4, leaf)[0]   # a power of two: nothing is rounded

    unit = gradient(True, True)
    assert torch.equal(gradient(True, False), unit * 4) and torch.equal(gradient(False, False), unit * 4)
    assert torch.equal(gradient(False, True), unit)


@pytest.mark.gpu
def test_a_traced_cross_entropy_is_refused():
    """What torch.jit.trace records of a function that overwrites its input does not run."""
    from aws_ofi_nccl_b200.ops import llm

    targets = torch.arange(6, device="cuda")
    traced = torch.jit.trace(lambda x: llm.cross_entropy(x * 1.0, targets), (torch.randn(6, 64, device="cuda").bfloat16(),), check_trace=False)
    with pytest.raises(RuntimeError, match="JIT"):
        traced(torch.randn(6, 64, device="cuda").bfloat16())
