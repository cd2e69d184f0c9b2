"""Kernels that start while the one before them ends: a chain of them, each reading what the one before has just written into
buffers that are used again and again, gives the same bits as one that is waited for after every call."""
import ctypes
import shutil
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu


class _Chain:
    """Optimizer step, residual norm, gate | up product, SwiGLU, split-K product back, cross entropy and the gradients of the
    products, all into buffers of its own."""

    def __init__(self, T, H, F):
        g = torch.Generator(device="cuda").manual_seed(T + H + F)

        def rnd(*s, std=1.0, dtype=torch.bfloat16):
            return (torch.randn(*s, device="cuda", generator=g) * std).to(dtype)

        self.T, self.H, self.F = T, H, F
        self.x, self.res, self.w = rnd(T, H), rnd(T, H), rnd(H, std=0.1) + 1
        self.wgu, self.wdown = rnd(2 * F, H, std=H ** -0.5), rnd(H, F, std=F ** -0.5)
        self.grad, self.m, self.v = torch.zeros_like(self.wgu), torch.zeros(2 * F, H, device="cuda"), torch.zeros(2 * F, H, device="cuda")
        self.targets = torch.randint(0, H, (T,), device="cuda", generator=g)
        self.buf = {k: torch.zeros(*s, device="cuda", dtype=d) for k, (s, d) in {
            "h": ((T, H), torch.bfloat16), "y": ((T, H), torch.bfloat16), "rstd": ((T,), torch.float32),
            "gu": ((T, 2 * F), torch.bfloat16), "act": ((T, F), torch.bfloat16), "out": ((T, H), torch.bfloat16),
            "loss": ((T,), torch.float32), "dact": ((T, F), torch.bfloat16), "dgu": ((T, 2 * F), torch.bfloat16),
            "dw": ((2 * F, H), torch.bfloat16), "q": ((T, F), torch.uint8), "qs": ((T,), torch.float32)}.items()}

    def steps(self):
        from aws_ofi_nccl_b200.ops import _lib
        from aws_ofi_nccl_b200.ops.gemm import gemm
        from aws_ofi_nccl_b200.ops.llm import adamw_step

        L, b, T, H, F = _lib.load(), self.buf, self.T, self.H, self.F

        def call(name, *args):
            _lib.check(getattr(L, name)(*[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args], _lib.stream_ptr()), name)

        yield lambda: adamw_step(self.wgu, self.grad, self.m, self.v, None, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8,
                                 weight_decay=0.1, step=3)
        yield lambda: call("b200_rmsnorm_fwd", self.x, self.res, b["h"], self.w, b["y"], b["rstd"], T, H, 1e-5)
        yield lambda: gemm(b["y"], self.wgu, out=b["gu"])
        yield lambda: call("b200_swiglu_fwd", b["gu"], b["act"], T, F)
        yield lambda: call("b200_quant_rows_fp8", b["act"], b["q"], b["qs"], T, F, F, F)
        yield lambda: gemm(b["act"], self.wdown, out=b["out"])
        yield lambda: call("b200_cross_entropy", b["out"], self.targets, b["loss"], T, H, H, 1.0 / T)
        yield lambda: gemm(b["out"], self.wdown, b_mn=True, out=b["dact"])
        yield lambda: call("b200_swiglu_bwd", b["dact"], b["gu"], b["dgu"], T, F)
        yield lambda: gemm(b["dgu"], b["y"], a_mn=True, b_mn=True, out=b["dw"])
        yield lambda: self.grad.copy_(b["dw"])   # what the next pass's optimizer step reads

    def run(self, wait):
        for step in self.steps():
            step()
            if wait:
                torch.cuda.synchronize()

    def results(self):
        return [t.clone() for t in (self.wgu, self.m, *self.buf.values())]


# less than a wave of everything; several waves; a long reduction that is split over clusters
@pytest.mark.parametrize("T,H,F", [(64, 128, 256), (1000, 1032, 2056), (128, 512, 8192), (4096, 2048, 4096)])
def test_a_chain_of_kernels_sees_what_the_kernel_before_wrote(T, H, F):
    waited, chained = _Chain(T, H, F), _Chain(T, H, F)
    for _ in range(3):
        waited.run(True)
    for _ in range(3):
        chained.run(False)
    for a, b in zip(waited.results(), chained.results()):
        assert torch.equal(a, b)


@pytest.mark.parametrize("T,H,F", [(64, 128, 256), (1000, 1032, 2056)])
def test_a_captured_chain_does_too(T, H, F):
    waited, captured = _Chain(T, H, F), _Chain(T, H, F)
    captured.run(False)   # what a first call sets up is no part of a graph
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=stream):
        captured.run(False)
    for _ in range(2):
        graph.replay()
    for _ in range(3):
        waited.run(True)
    torch.cuda.synchronize()
    for a, b in zip(waited.results(), captured.results()):
        assert torch.equal(a, b)


class _Layers:
    """Embedding, residual norm, projection, rotary split, a wide head's cross entropy, and what leads back from there: rotary split, projection, norm
    with its weight's gradient, embedding. No id comes twice, so that the table's gradient is the same every time."""

    def __init__(self, T, heads, hd, V):
        g = torch.Generator(device="cuda").manual_seed(T + heads + V)
        bf, f32 = torch.bfloat16, torch.float32

        def rnd(*s, std=1.0):
            return (torch.randn(*s, device="cuda", generator=g) * std).to(bf)

        H, P = heads * hd, (heads + 2) * hd
        self.T, self.heads, self.hd, self.V, self.H, self.P = T, heads, hd, V, H, P
        self.ids, self.targets = torch.randperm(2 * T, device="cuda", generator=g)[:T], torch.randint(0, V, (T,), device="cuda", generator=g)
        self.table, self.res, self.w = rnd(2 * T, H), rnd(T, H), rnd(H, std=0.1) + 1
        self.wqkv, self.head = rnd(P, H, std=H ** -0.5), rnd(V, H, std=H ** -0.5)
        self.cos, self.sin = torch.rand(T, hd // 2, device="cuda", generator=g), torch.rand(T, hd // 2, device="cuda", generator=g)
        self.buf = {k: torch.zeros(*shape, device="cuda", dtype=d) for k, (shape, d) in {
            "x": ((T, H), bf), "h": ((T, H), bf), "y": ((T, H), bf), "rstd": ((T,), f32), "qkv": ((T, P), bf), "q": ((T, H), bf), "k": ((T, hd), bf),
            "v": ((T, hd), bf), "logits": ((T, V), bf), "loss": ((T,), f32), "dy": ((T, H), bf), "dqkv": ((T, P), bf), "dn": ((T, H), bf),
            "dx": ((T, H), bf), "dw": ((H,), bf), "dtable": ((2 * T, H), bf)}.items()}

    def steps(self):
        from aws_ofi_nccl_b200.ops import _lib
        from aws_ofi_nccl_b200.ops.gemm import gemm

        L, b, T, H = _lib.load(), self.buf, self.T, self.H
        partial = self.buf.setdefault("partial", torch.zeros(L.b200_rmsnorm_bwd_partial_rows(), H, device="cuda"))
        strides = (ctypes.c_longlong * 9)(*[n for row in (H, self.hd, self.hd) for n in (0, row, self.hd)])

        def call(name, *args):
            fn = getattr(L, name)
            _lib.check(fn(*[ctypes.c_void_p(a.data_ptr()) if isinstance(a, torch.Tensor) else a for a in args], ctypes.c_void_p(_lib.stream_ptr())), name)

        def rope(qkv, backward):
            call("b200_rope_qkv", qkv, ctypes.c_longlong(self.P), b["q"], b["k"], b["v"], strides, self.cos, self.sin, ctypes.c_longlong(T), self.heads, 1, self.hd, T, backward)

        yield lambda: call("b200_embedding_fwd", self.ids, self.table, b["x"], T, H)
        yield lambda: call("b200_rmsnorm_fwd", b["x"], self.res, b["h"], self.w, b["y"], b["rstd"], T, H, 1e-5)
        yield lambda: gemm(b["y"], self.wqkv, out=b["qkv"])
        yield lambda: rope(b["qkv"], 0)
        yield lambda: gemm(b["y"], self.head, out=b["logits"])
        yield lambda: call("b200_cross_entropy", b["logits"], self.targets, b["loss"], T, self.V, self.V, 1.0)
        yield lambda: gemm(b["logits"], self.head, b_mn=True, out=b["dy"])
        yield lambda: rope(b["dqkv"], 1)
        yield lambda: gemm(b["dqkv"], self.wqkv, b_mn=True, out=b["dn"])
        yield lambda: call("b200_rmsnorm_bwd", b["dn"], b["h"], self.w, b["rstd"], b["dy"], b["dx"], partial, b["dw"], 0, T, H)
        yield lambda: call("b200_embedding_bwd", self.ids, b["dx"], b["dtable"], T, H)
        yield lambda: self.table.copy_(b["dtable"])   # what the next pass looks up

    run = _Chain.run

    def run_on(self, streams):
        """Each kernel on the other stream than the one before, behind it and behind the one before that."""
        streams[1].wait_stream(streams[0])
        for i, step in enumerate(self.steps()):
            here, other = streams[i % 2], streams[1 - i % 2]
            here.wait_stream(other)
            with torch.cuda.stream(here):
                step()
        streams[0].wait_stream(streams[1])

    def results(self):
        return [t.clone() for t in (self.table, *self.buf.values())]


# tokens that fill no wave; norms through rings and streamed rows of the head
LAYERS = [(64, 4, 64, 1000), (1000, 16, 128, 2056), (300, 4, 128, 32776)]


@pytest.mark.parametrize("T,heads,hd,V", LAYERS)
def test_a_chain_of_layers_does_too(T, heads, hd, V):
    waited, chained = _Layers(T, heads, hd, V), _Layers(T, heads, hd, V)
    for _ in range(3):
        waited.run(True)
    for _ in range(3):
        chained.run(False)
    for a, b in zip(waited.results(), chained.results()):
        assert torch.equal(a, b)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("T,heads,hd,V", LAYERS)
def test_and_a_chain_over_two_streams(T, heads, hd, V, captured):
    """A kernel behind one on its own stream and one on another waits for both."""
    waited, chained = _Layers(T, heads, hd, V), _Layers(T, heads, hd, V)
    for _ in range(3):
        waited.run(True)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    if captured:
        chained.run(False)   # what a first call sets up is no part of a graph
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            chained.run_on(streams)
        for _ in range(2):
            graph.replay()
    else:
        for _ in range(3):
            chained.run_on(streams)
    torch.cuda.synchronize()
    for a, b in zip(waited.results(), chained.results()):
        assert torch.equal(a, b)


FIRST_CALL = """
import torch
from aws_ofi_nccl_b200.ops import _lib
from aws_ofi_nccl_b200.ops.gemm import gemm
bf = dict(device="cuda", dtype=torch.bfloat16)
x, y, w, rstd = torch.ones(%(T)d, %(W)d, **bf), torch.zeros(%(T)d, %(W)d, **bf), torch.ones(%(W)d, **bf), torch.zeros(%(T)d, device="cuda")
targets, loss, sq = torch.zeros(%(T)d, device="cuda", dtype=torch.int64), torch.zeros(%(T)d, device="cuda"), torch.zeros(%(T)d, %(T)d, **bf)
lib, p = _lib.load(), lambda t: t.data_ptr()
calls = {
    "norm": lambda s: lib.b200_rmsnorm_fwd(p(x), None, None, p(w), p(y), p(rstd), %(T)d, %(W)d, 0.0, s),
    "cross_entropy": lambda s: lib.b200_cross_entropy(p(x), p(targets), p(loss), %(T)d, %(W)d, %(W)d, 1.0, s),
    "product": lambda s: int(gemm(x, x, out=sq) is not sq),
}
torch.cuda.synchronize()
stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream):
    assert calls["%(name)s"](stream.cuda_stream) == 0
graph.replay()
torch.cuda.synchronize()
result = {"norm": y, "cross_entropy": loss, "product": sq}["%(name)s"]
want = {"norm": 1.0, "cross_entropy": torch.tensor(%(W)d, dtype=torch.float64).log().item(), "product": %(W)d}["%(name)s"]
assert ((result.double() - want).abs() <= 2.0 ** -8 * want).all(), result
assert _lib.read_status() == 0
"""


# rows that come through rings of shared memory, and a product
@pytest.mark.parametrize("name,T,W", [("norm", 2400, 8192), ("cross_entropy", 300, 32776), ("product", 512, 256)])
def test_a_process_whose_first_call_is_captured(name, T, W):
    r = subprocess.run([sys.executable, "-c", FIRST_CALL % {"name": name, "T": T, "W": W}], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parent.parent)
    assert r.returncode == 0, r.stderr[-3000:]


def test_two_copies_of_the_library_in_one_process(tmp_path):
    """Each raises the limits of its own kernels."""
    from aws_ofi_nccl_b200.ops import _lib

    copy = tmp_path / "copy.so"
    shutil.copyfile(_lib.lib_path(), copy)
    second, ll, vp = ctypes.CDLL(str(copy)), ctypes.c_longlong, lambda t: ctypes.c_void_p(t.data_ptr())
    x = torch.ones(512, 256, device="cuda", dtype=torch.bfloat16)
    for lib in (_lib.load(), second):
        out = torch.zeros(512, 512, device="cuda", dtype=torch.bfloat16)
        assert lib.b200_gemm_bf16(vp(x), vp(x), vp(out), 512, 512, 256, ll(256), ll(256), ll(512), 0, 0, 0, 0, 0, 0, ctypes.c_void_p(_lib.stream_ptr())) == 0
        assert (out == 256).all()


def _programmatic(calls):
    """Of kernels captured one after the other: whether each after the first may come up before the one before it has ended."""
    graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        for call in calls:
            call()
    driver, raw, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(len(calls))
    start, to, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (ctypes.c_uint8 * 8 * n.value)()
    assert driver.cuGraphGetEdges_v2(raw, start, to, data, ctypes.byref(n)) == 0 and n.value == len(calls) - 1
    after = {a: (b, kind[2] == 1) for a, b, kind in zip(start, to, data) if a}   # ports of both ends, then the edge's type
    at, = set(after) - {b for b, _ in after.values()}
    out = []
    while at in after:
        at, early = after[at]
        out.append(early)
    return out


@pytest.mark.parametrize("M,N", [(512, 1024), (128, 512)])   # CTA pairs, single CTAs
def test_a_product_that_leaves_room_is_launched_when_the_kernel_before_has_ended(M, N):
    from aws_ofi_nccl_b200.ops.gemm import gemm

    a, b, out = (torch.zeros(*s, device="cuda", dtype=torch.bfloat16) for s in ((M, 256), (N, 256), (M, N)))
    product = [lambda c=c: gemm(a, b, out=out, max_ctas=c) for c in (0, 0, 100, 100, 2, 148, 0)]
    product[0]()   # what a first call sets up
    assert _programmatic(product) == [True, False, False, False, True, True]


def test_room_that_a_product_leaves_is_there_for_another_stream():
    """Products on 74 SMs beside a chain of products that leaves these free take about as long as by themselves (16 us, 72 beside
    a chain that leaves none)."""
    from aws_ofi_nccl_b200.ops.gemm import gemm

    big, small = (torch.randn(n, n, device="cuda").bfloat16() for n in (2048, 1024))
    outs = [torch.empty_like(big), torch.empty_like(small)]
    chain, side = torch.cuda.Stream(), torch.cuda.Stream()

    def times(products):
        events = [[torch.cuda.Event(enable_timing=True) for _ in range(2)] for _ in range(40)]
        torch.cuda._sleep(4_000_000)   # everything is queued before anything runs
        for s in (chain, side):
            s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(chain):
            for _ in range(products):
                gemm(big, big, out=outs[0], max_ctas=74)
        with torch.cuda.stream(side):
            for begin, end in events:
                begin.record()
                gemm(small, small, out=outs[1], max_ctas=74)
                end.record()
        torch.cuda.synchronize()
        return sorted(b.elapsed_time(e) for b, e in events)

    times(1)
    alone, beside = times(0), times(60)
    assert beside[20] < 2 * alone[20] and beside[-1] < 3 * alone[20]
    assert all(torch.equal(o, gemm(x, x)) for o, x in zip(outs, (big, small)))
