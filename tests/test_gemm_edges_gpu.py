"""Products with few output tiles and a long reduction (cluster split-K) and the edges of the stored
tiles, against a product in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

# one 128-row tile / ragged rows and columns; single CTAs and 256-row tiles on CTA pairs; K with a tail
SPLIT = [(1, 8, 4096), (128, 4096, 14336), (130, 264, 8200), (256, 128, 4096), (300, 520, 8248), (512, 768, 16384), (1000, 1000, 8200)]
# no split: edges of the 64-column and 32-row slabs that the epilogue stores
WHOLE = [(16, 72, 2056), (33, 72, 64), (129, 200, 136), (257, 328, 72), (2000, 1032, 128)]


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", SPLIT + WHOLE)
def test_product_and_accumulation(M, N, K, out_dtype, a_mn, b_mn):
    from aws_ofi_nccl_b200.ops.gemm import gemm

    if a_mn:
        M = (M + 7) // 8 * 8   # the pitch of a transposed operand is a multiple of 16 bytes
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda", generator=g).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda", generator=g).bfloat16()
    A, B = (a.T if a_mn else a).double(), (b if b_mn else b.T).double()
    ref, mag = A @ B, A.abs() @ B.abs()
    # the output lies in a larger buffer whose other elements must stay as they were
    pad = torch.full((M + 1, (N + 15) // 8 * 8), 7.0, device="cuda", dtype=out_dtype)
    out = pad[:M, :N]
    step = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -24
    # fp32 sums of K exact products in any order: K ulp of the sum of their magnitudes, far from reached
    bound = K * 2.0 ** -24 * mag + step * ref.abs()
    gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out)
    assert ((out.double() - ref).abs() <= bound).all()
    first = out.double()
    gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=True)
    want = first + ref
    assert ((out.double() - want).abs() <= bound + step * want.abs() + 2.0 ** -24 * (first.abs() + mag)).all()
    assert (pad[M:] == 7).all() and (pad[:, N:] == 7).all()


# groups of M tiles where both operands are small; beside a larger one all M tiles of a column before the next column, or all N tiles of a row before the
# next row; the last wave halved or not
@pytest.mark.parametrize("M,N,K", [(2504, 2632, 72), (2632, 2504, 72), (2312, 4104, 200), (4104, 2312, 200), (2504, 15008, 520), (15008, 2504, 520),
                                   (2312, 8200, 1000), (8200, 2312, 1000)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_every_tile_is_computed_in_either_order_of_tiles(M, N, K, b_mn):
    from aws_ofi_nccl_b200.ops.gemm import gemm

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), device="cuda", generator=g).bfloat16()
    A, B = a.double(), (b if b_mn else b.T).double()
    ref, out = A @ B, torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(a, b, b_mn=b_mn, out=out)
    # K products in fp32 in any order, rounded once to bf16
    assert ((out.double() - ref).abs() <= K * 2.0 ** -24 * (A.abs() @ B.abs()) + 2.0 ** -8 * ref.abs()).all()


def _plan(M, N, K, a_mn=False, b_mn=False):
    """(pair, tile width, slices) of the automatic choice."""
    from aws_ofi_nccl_b200.ops import _lib

    out = [ctypes.c_int() for _ in range(3)]
    lda, ldb = ctypes.c_longlong(M if a_mn else K), ctypes.c_longlong(N if b_mn else K)
    assert _lib.load().b200_gemm_plan(M, N, K, lda, ldb, *(ctypes.byref(o) for o in out)) == 0
    return tuple(o.value for o in out)


def test_the_listed_sizes_take_the_path_that_they_are_listed_for():
    assert all(_plan(*s)[2] > 1 for s in SPLIT) and all(_plan(*s)[2] == 1 for s in WHOLE)
    assert {_plan(*s)[::2] for s in SPLIT} == {(0, 4), (0, 8), (1, 2), (1, 4)}


@pytest.mark.parametrize("M,N,K", [(257, 4744, 200), (384, 6144, 72), (300, 6272, 1032)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_three_rows_of_tiles_that_all_run_at_once(M, N, K, a_mn, b_mn):
    assert _plan(M, N, K) == (0, 128, 1)
    test_product_and_accumulation(M, N, K, torch.bfloat16, a_mn, b_mn)


@pytest.mark.parametrize("M,N", [(256, 6144), (385, 6144), (384, 4736), (384, 6280)])
def test_other_rows_and_columns_stay_on_pairs(M, N):
    assert _plan(M, N, 2048)[0] == 1


def test_products_on_single_ctas_have_no_pair_tiles():
    """Nor do they change what SwiGLU's products run on, whose epilogues need the sums in 32 bits."""
    from aws_ofi_nccl_b200.ops import _lib

    lib, ll, vp = _lib.load(), ctypes.c_longlong, ctypes.c_void_p
    w, h = ctypes.c_int(), ctypes.c_int()
    for M, N, want in ((300, 6144, 10001), (256, 6144, 0), (385, 6144, 0), (128, 6144, 10001)):
        assert lib.b200_gemm_tiles(M, N, 2048, ll(2048), ll(2048), 0, ctypes.byref(w), ctypes.byref(h)) == want
    assert lib.b200_gemm_swiglu_launches(vp(4096), vp(4096), 300, 3072, 2048, ll(2048)) == 1
    assert lib.b200_gemm_swiglu_bwd_launches(vp(4096), vp(4096), 300, 6144, 2048, ll(6144)) == 1


@pytest.mark.parametrize("M,N,K", [(256, 256, 1024), (512, 1024, 2048), (128, 4096, 1024), (768, 1536, 2048)])
def test_a_short_reduction_is_not_split(M, N, K):
    """Products that a split made up to 1.4 times slower."""
    assert _plan(M, N, K)[2] == 1


@pytest.mark.parametrize("M,N,K", [(6, 560, 1392), (24, 560, 2032), (67, 304, 1272), (8, 2784, 2528), (198, 288, 2600)])
def test_few_rows_and_a_reduction_that_is_worth_splitting(M, N, K):
    """Products of single CTAs whose narrow tiles need no more waves than wide ones, and that are faster split: by 1.2 to 1.6 times."""
    assert _plan(M, N, K)[2] > 1


@pytest.mark.parametrize("M,N,K", [(16, 624, 256), (4, 288, 1112), (35, 408, 1192), (33, 1632, 760)])
def test_few_rows_and_a_short_reduction_take_narrow_tiles(M, N, K):
    """0.67 to 0.85 of the time of wide ones."""
    assert _plan(M, N, K) == (0, 128, 1)


@pytest.mark.parametrize("M,N,K,wide", [(1068, 3832, 6432, False), (744, 8592, 2336, False),   # rows on 64 bytes
                                        (1000, 5160, 2568, True), (4096, 4096, 16040, True),     # rows anywhere
                                        (4096, 4096, 14336, False), (6286, 2368, 640, True)])    # rows on cache lines
def test_tile_width_follows_how_the_rows_lie(M, N, K, wide):
    assert _plan(M, N, K) == (1, 256 if wide else 128, 1)


@pytest.mark.parametrize("pair,slices", [(0, 2), (0, 4), (0, 8), (1, 2), (1, 4)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_every_split_kernel(pair, slices, a_mn, b_mn, out_dtype):
    """Each member, major and output, asked for by name: ragged rows, columns and K, fewer blocks of K than
    a slice's pipeline has stages, one block per slice."""
    from aws_ofi_nccl_b200.ops import _lib

    ll = ctypes.c_longlong
    step = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -24
    for M, N, K in ((8, 16, 64 * slices), (264, 200, 1096), (520, 136, 2056)):
        g = torch.Generator(device="cuda").manual_seed(M + slices)
        a = torch.randn((K, M) if a_mn else (M, K), device="cuda", generator=g).bfloat16()
        b = torch.randn((K, N) if b_mn else (N, K), device="cuda", generator=g).bfloat16()
        A, B = (a.T if a_mn else a).double(), (b if b_mn else b.T).double()
        ref, mag = A @ B, A.abs() @ B.abs()
        pad = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=out_dtype)
        want = torch.zeros_like(ref)
        for accumulate in (0, 1):
            rc = _lib.load().b200_gemm_bf16_split(
                ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(pad.data_ptr()), M, N, K,
                ll(a.stride(0)), ll(b.stride(0)), ll(pad.stride(0)), int(a_mn), int(b_mn), int(out_dtype == torch.float32), accumulate,
                pair, slices, ctypes.c_void_p(_lib.stream_ptr()))
            assert rc == 0
            want = want + ref
            # fp32 sums of K exact products in any order, one rounding of the output
            bound = K * 2.0 ** -24 * mag + 2 * step * want.abs()
            assert ((pad[:M, :N].double() - want).abs() <= bound).all()
            want = pad[:M, :N].double()
        assert (pad[M:] == 7).all() and (pad[:, N:] == 7).all()


def test_split_sums_are_the_same_every_time_and_on_two_streams():
    from aws_ofi_nccl_b200.ops.gemm import gemm

    a = torch.randn(128, 14336, device="cuda").bfloat16()
    b = torch.randn(4096, 14336, device="cuda").bfloat16()
    want = gemm(a, b)
    torch.cuda.synchronize()
    streams, outs = [torch.cuda.Stream() for _ in range(2)], []
    for i in range(6):
        with torch.cuda.stream(streams[i % 2]):
            outs.append(gemm(a, b))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)


@pytest.mark.parametrize("M,N,K", [(256, 128, 128), (300, 200, 144), (257, 1000, 272)])
def test_fp8_product_at_ragged_edges(M, N, K):
    from aws_ofi_nccl_b200.ops.gemm import gemm_fp8, quantize_rows_fp8

    xq, xs = quantize_rows_fp8(torch.randn(M, K, device="cuda").bfloat16())
    wq, ws = quantize_rows_fp8(torch.randn(N, K, device="cuda").bfloat16())
    X, W = xq.double() * xs.double()[:, None], wq.double() * ws.double()[:, None]
    ref, mag = X @ W.T, X.abs() @ W.T.abs()
    out = gemm_fp8(xq, wq, xs, ws)
    # bf16 rounding of the result, two fp32 roundings of the scales, fp32 sums
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (K + 4) * 2.0 ** -24 * mag).all()


def _padded(rows, cols, g):
    """A [rows, cols] matrix whose pitch is a multiple of 16 bytes."""
    return torch.randn(rows, (cols + 7) // 8 * 8, device="cuda", generator=g).bfloat16()[:, :cols]


@pytest.mark.parametrize("split", [0, 2, 4])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(5, 3, 264), (129, 130, 517), (258, 133, 263), (300, 257, 520), (1030, 389, 261)])
def test_widths_that_are_no_multiple_of_a_vector(M, N, K, out_dtype, a_mn, b_mn, split):
    """The stores end in the middle of a 16-byte vector, and nothing beyond is touched."""
    from aws_ofi_nccl_b200.ops import _lib
    from aws_ofi_nccl_b200.ops.gemm import gemm

    ll, vp = ctypes.c_longlong, ctypes.c_void_p
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = _padded(*((K, M) if a_mn else (M, K)), g), _padded(*((K, N) if b_mn else (N, K)), g)
    A, B = (a.T if a_mn else a).double(), (b if b_mn else b.T).double()
    ref, mag = A @ B, A.abs() @ B.abs()
    pad = torch.full((M + 1, (N + 15) // 8 * 8), 7.0, device="cuda", dtype=out_dtype)
    out = pad[:M, :N]
    step = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -24
    want = torch.zeros_like(ref)
    for accumulate in (False, True):
        if split:
            rc = _lib.load().b200_gemm_bf16_split(
                vp(a.data_ptr()), vp(b.data_ptr()), vp(out.data_ptr()), M, N, K, ll(a.stride(0)), ll(b.stride(0)),
                ll(out.stride(0)), int(a_mn), int(b_mn), int(out_dtype == torch.float32), int(accumulate), int(M >= 256 and N >= 128),
                split, vp(_lib.stream_ptr()))
            assert rc == 0
        else:
            gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=accumulate)
        want = want + ref
        # fp32 sums of K exact products in any order, one rounding of the output
        assert ((out.double() - want).abs() <= K * 2.0 ** -24 * mag + 2 * step * want.abs()).all()
        want = out.double()
    assert (pad[M:] == 7).all() and (pad[:, N:] == 7).all()


@pytest.mark.parametrize("M,N,K", [(256, 132, 128), (257, 300, 272), (515, 260, 144)])
def test_fp8_widths_that_are_no_multiple_of_a_vector(M, N, K):
    from aws_ofi_nccl_b200.ops.gemm import gemm_fp8, quantize_rows_fp8

    xq, xs = quantize_rows_fp8(torch.randn(M, K, device="cuda").bfloat16())
    wq, ws = quantize_rows_fp8(torch.randn(N, K, device="cuda").bfloat16())
    X, W = xq.double() * xs.double()[:, None], wq.double() * ws.double()[:, None]
    ref, mag = X @ W.T, X.abs() @ W.T.abs()
    pad = torch.full((M + 1, (N + 15) // 8 * 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm_fp8(xq, wq, xs, ws, out=pad[:M, :N])
    # bf16 rounding of the result, two fp32 roundings of the scales, fp32 sums
    assert ((pad[:M, :N].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (K + 4) * 2.0 ** -24 * mag).all()
    assert (pad[M:] == 7).all() and (pad[:, N:] == 7).all()


@pytest.mark.parametrize("width,halves", [(128, 0), (160, 0), (192, 0), (224, 0), (256, 0), (256, 1)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_every_tile_width_and_the_halved_last_wave(width, halves, out_dtype, a_mn, b_mn):
    """Tiles that end inside a 64-column slab, beside others and at the last column; rows, columns and K that fill
    no tile; one tile and 126 of them (74 whole ones and a last wave whose halves may lie beyond the last column)."""
    from aws_ofi_nccl_b200.ops import _lib

    ll, vp = ctypes.c_longlong, ctypes.c_void_p
    step = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -24
    for M, N, K in ((256, 128, 64), (296, 333, 200), (512, 1027, 72), (2304, 3330, 136)):
        g = torch.Generator(device="cuda").manual_seed(M + width)
        a, b = _padded(*((K, M) if a_mn else (M, K)), g), _padded(*((K, N) if b_mn else (N, K)), g)
        A, B = (a.T if a_mn else a).double(), (b if b_mn else b.T).double()
        ref, mag = A @ B, A.abs() @ B.abs()
        pad = torch.full((M + 1, (N + 15) // 8 * 8), 7.0, device="cuda", dtype=out_dtype)
        want = torch.zeros_like(ref)
        for accumulate in (0, 1):
            rc = _lib.load().b200_gemm_bf16_tiles(
                vp(a.data_ptr()), vp(b.data_ptr()), vp(pad.data_ptr()), M, N, K, ll(a.stride(0)), ll(b.stride(0)),
                ll(pad.stride(0)), int(a_mn), int(b_mn), int(out_dtype == torch.float32), accumulate, width, halves,
                vp(_lib.stream_ptr()))
            assert rc == 0
            want = want + ref
            # fp32 sums of K exact products in any order, one rounding of the output
            assert ((pad[:M, :N].double() - want).abs() <= K * 2.0 ** -24 * mag + 2 * step * want.abs()).all()
            want = pad[:M, :N].double()
        assert (pad[M:] == 7).all() and (pad[:, N:] == 7).all()


@pytest.mark.parametrize("K", [8, 192, 200])
@pytest.mark.parametrize("M,N", [(500, 37 * 256), (512, 37 * 256 + 8), (1, 8)])
def test_a_tile_for_every_pair_and_one_more(M, N, K):
    """74 wide tiles, as many as there are pairs of CTAs, then 76 of them, and a single one: the epilogue's warps differ."""
    from aws_ofi_nccl_b200.ops import _lib

    ll, vp = ctypes.c_longlong, ctypes.c_void_p
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    pad = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    rc = _lib.load().b200_gemm_bf16_tiles(vp(a.data_ptr()), vp(b.data_ptr()), vp(pad.data_ptr()), M, N, K, ll(K), ll(K), ll(N + 8),
                                          0, 0, 0, 0, 256, 0, vp(_lib.stream_ptr()))
    assert rc == 0
    ref, mag = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    # fp32 sums of K exact products in any order, one rounding of the output
    assert ((pad[:M, :N].double() - ref).abs() <= K * 2.0 ** -24 * mag + 2.0 ** -8 * ref.abs()).all()
    assert (pad[M:] == 7).all() and (pad[:, N:] == 7).all()


def _tiles(M, N, K, b_mn=False):
    """(width, halves) that the automatic choice runs on, for operands with contiguous rows."""
    from aws_ofi_nccl_b200.ops import _lib

    w, h = ctypes.c_int(), ctypes.c_int()
    ll = ctypes.c_longlong
    assert _lib.load().b200_gemm_tiles(M, N, K, ll(K), ll(N if b_mn else K), int(b_mn), ctypes.byref(w), ctypes.byref(h)) == 0
    return w.value, h.value


@pytest.mark.parametrize("M,N,K,b_mn,want", [
    (4096, 4096, 4096, False, (256, 1)), (4096, 14336, 4096, False, (256, 1)), (4096, 28672, 4096, True, (256, 1)),
    (384, 10736, 3712, False, (160, 0)), (1280, 7744, 328, False, (192, 0)),
    (1000, 2568, 5160, False, (160, 0)), (1000, 2568, 5160, True, (256, 0)),   # rows off cache lines
    (768, 256, 768, False, (128, 0)), (1920, 4280, 824, False, (256, 0))])
def test_tiles_follow_the_waves_that_they_fill(M, N, K, b_mn, want):
    """Choices that were measured to be the faster ones."""
    assert _tiles(M, N, K, b_mn) == want


@pytest.mark.parametrize("M,N,K,b_mn,want", [
    (768, 8192, 8192, False, (192, 0)), (768, 8192, 4096, True, (192, 0)), (768, 8192, 4032, False, (256, 1)),
    (768, 8192, 8200, False, (256, 1)),   # rows off cache lines
    (2403, 7680, 11456, False, (224, 0)), (2403, 7680, 2304, False, (256, 1))])
def test_a_long_reduction_halves_fewer_waves(M, N, K, b_mn, want):
    """Choices that were measured to be the faster ones, on both sides of where they change."""
    assert _tiles(M, N, K, b_mn) == want


@pytest.mark.parametrize("M,N,K", [(4096, 2072, 256), (2304, 3332, 144), (513, 300, 272)])
def test_fp8_product_on_every_kind_of_tile(M, N, K):
    """A last wave of halves, a ragged width, single tiles."""
    from aws_ofi_nccl_b200.ops.gemm import gemm_fp8, quantize_rows_fp8

    xq, xs = quantize_rows_fp8(torch.randn(M, K, device="cuda").bfloat16())
    wq, ws = quantize_rows_fp8(torch.randn(N, K, device="cuda").bfloat16())
    X, W = xq.double() * xs.double()[:, None], wq.double() * ws.double()[:, None]
    ref, mag = X @ W.T, X.abs() @ W.T.abs()
    pad = torch.full((M + 1, (N + 15) // 8 * 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm_fp8(xq, wq, xs, ws, out=pad[:M, :N])
    # bf16 rounding of the result, two fp32 roundings of the scales, fp32 sums
    assert ((pad[:M, :N].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (K + 4) * 2.0 ** -24 * mag).all()
    assert (pad[M:] == 7).all() and (pad[:, N:] == 7).all()
