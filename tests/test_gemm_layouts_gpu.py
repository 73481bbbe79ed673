"""16-bit products by the layout of their operands: extents of 1, rows on and off the 16-byte grid, strides in either order."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DT = {"f16": torch.float16, "bf16": torch.bfloat16}
UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}


def close(got, want, k, magnitude):
    """One rounding of the result and the fp32 sum's error: k additions of at most `magnitude` (the sum of the absolute products)."""
    assert got.shape == want.shape
    bound = UNIT[got.dtype] * want.abs() + k * 2.0 ** -24 * magnitude + 2.0 ** -24
    worst = ((got.double() - want).abs() / bound).max().item()
    assert worst <= 1.0, worst


def product(a, b, dt):
    return a.double() @ b.double(), a.double().abs() @ b.double().abs()


# above and below 32 768 and 65 536 multiplications, where the dispatch changes
@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("m,n,k", [(512, 512, 1), (4096, 77, 1), (100, 1000, 1), (1, 4096, 64), (1, 1001, 129), (4096, 1, 64), (1001, 1, 129), (1, 1, 70000),
                                   (1, 65544, 1), (65543, 1, 1), (2, 3, 11000), (33, 31, 63), (64, 64, 8)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (True, False), (False, True), (True, True)])
def test_extents_of_one(m, n, k, trans_a, trans_b, dt):
    from metalhlo_b200 import cuda

    g = torch.Generator().manual_seed(m + n + k)
    a, b = torch.randn(m, k, generator=g).to(DT[dt]).cuda(), (torch.randn(k, n, generator=g) / math.sqrt(k)).to(DT[dt]).cuda()
    got = cuda.gemm(a.t().contiguous() if trans_a else a, b.t().contiguous() if trans_b else b, trans_a=trans_a, trans_b=trans_b)
    close(got, *product(a, b, dt)[:1], k, product(a, b, dt)[1])


@pytest.mark.parametrize("m,n,k", [(512, 512, 1), (300, 1001, 1), (1, 4096, 33), (2049, 1, 65)])
@pytest.mark.parametrize("ca,cb", [(1, 0), (0, 0), (1, 1), (0, 1)])
def test_extents_of_one_in_a_program(m, n, k, ca, cb):
    from metalhlo_b200 import capi
    from metalhlo_b200.modules import func, tt

    g = torch.Generator().manual_seed(7 * m + n)
    a, b = torch.randn(m, k, generator=g).half(), (torch.randn(k, n, generator=g) / math.sqrt(k)).half()
    sa, sb = ((m, k) if ca else (k, m)), ((n, k) if cb else (k, n))
    text = func([tt(sa, "f16"), tt(sb, "f16")], [tt((m, n), "f16")],
                f"    %0 = stablehlo.dot_general %arg0, %arg1, contracting_dims = [{ca}] x [{cb}] : ({tt(sa, 'f16')}, {tt(sb, 'f16')}) -> {tt((m, n), 'f16')}", "%0")
    got = torch.from_numpy(capi.Client().run(text, [(a if ca else a.t()).contiguous(), (b.t() if cb else b).contiguous()], opt_level=3)[0])
    close(got, *product(a, b, "f16")[:1], k, product(a, b, "f16")[1])


def strided(x, order, pitch, offset=0):
    """x [rows, cols] in a larger buffer: `order` "row" or "col" major with that pitch, or every second element ("both")."""
    rows, cols = x.shape
    if order == "both":
        buf = torch.zeros(offset + 2 * rows * pitch, dtype=x.dtype, device="cuda")
        view = buf[offset:].as_strided((rows, cols), (2 * pitch, 2))
    else:
        buf = torch.zeros(offset + (rows if order == "row" else cols) * pitch, dtype=x.dtype, device="cuda")
        view = buf[offset:].as_strided((rows, cols), (pitch, 1) if order == "row" else (1, pitch))
    view.copy_(x)
    return view


def raw_gemm(a, b, dtype, b0=1, b1=1, a_batch=(0, 0), b_batch=(0, 0), bias=None, epilogue="none", tuning=None, out_dtype=None):
    """mhlo_cuda_gemm_tuned on views: a [m, k], b [k, n]."""
    import ctypes as C

    from metalhlo_b200 import cuda

    (m, k), n = a.shape[-2:], b.shape[-1]
    out = torch.full((b0, b1, m, n), float("nan"), dtype=out_dtype or dtype, device="cuda")
    t = cuda.GemmTuning(*tuning) if tuning else None
    code = cuda.torch_dtype_code
    cuda.check(cuda.lib.mhlo_cuda_gemm_tuned(code(dtype), code(out.dtype), a.data_ptr(), cuda._i64s([*a_batch, *a.stride()[-2:]]), b.data_ptr(),
                                             cuda._i64s([*b_batch, *b.stride()[-2:]]), out.data_ptr(), b0, b1, m, n, k,
                                             None if bias is None else bias.data_ptr(), cuda.EPILOGUES[epilogue], C.byref(t) if t else None,
                                             torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out


# rows that start on the grid, rows that do not, a base that does not, the other order, no contiguous dimension; K of 1 on the grid
@pytest.mark.parametrize("m,n,k", [(300, 257, 65), (512, 512, 1), (1, 3000, 40), (3000, 1, 40)])
@pytest.mark.parametrize("la", [("row", 0, 0), ("row", 1, 0), ("row", 0, 1), ("col", 0, 0), ("col", 3, 0), ("both", 0, 0)])
@pytest.mark.parametrize("lb", [("row", 0, 0), ("row", 1, 0), ("col", 0, 0), ("col", 5, 2), ("both", 0, 0)])
def test_views(m, n, k, la, lb):
    g = torch.Generator().manual_seed(m)
    a, b = torch.randn(m, k, generator=g).half().cuda(), (torch.randn(k, n, generator=g) / math.sqrt(k)).half().cuda()
    views = []
    for x, (order, extra, offset) in ((a, la), (b, lb)):
        inner = x.shape[0] if order == "col" else x.shape[1]
        views.append(strided(x, order, (inner + 7) // 8 * 8 + extra, offset))
    want, magnitude = product(a, b, "f16")
    close(raw_gemm(*views, torch.float16)[0, 0], want, k, magnitude)


# packed; few results, read in place; K of 1; few results with K split over a cluster
ODD = [(65, 67, 69, 0), (300, 1001, 77, 0), (16, 128, 256, 0), (512, 512, 1, 0), (33, 96, 4096, 1), (129, 70, 515, 1)]


@pytest.mark.parametrize("m,n,k,split", ODD + [(512, 512, 64, 0), (512, 512, 512, 1)])
@pytest.mark.parametrize("out_dtype", [torch.float16, torch.float32])
def test_relu_hands_a_nan_on(m, n, k, split, out_dtype):
    g = torch.Generator().manual_seed(m)
    a, b = torch.randn(m, k, generator=g).half().cuda(), torch.randn(k, n, generator=g).half().cuda()
    a[m // 2, 0] = math.nan
    got = raw_gemm(a, b, torch.float16, epilogue="relu", tuning=(0, 0, 0, split), out_dtype=out_dtype)[0, 0]
    bad = torch.isnan(got)
    assert bool(bad[m // 2].all()) and int(bad.sum()) == n
    assert float(got[~bad].min()) == 0.0


ACT = {"gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh"), "gelu_erf": torch.nn.functional.gelu,
       "silu": torch.nn.functional.silu, "tanh": torch.tanh, "sigmoid": torch.sigmoid, "relu": torch.relu}


@pytest.mark.parametrize("m,n,k,split", ODD)
@pytest.mark.parametrize("epilogue", sorted(ACT))
@pytest.mark.parametrize("dt,out_dtype", [("f16", torch.float16), ("bf16", torch.bfloat16), ("bf16", torch.float32)])
def test_activations_in_fp32(m, n, k, split, epilogue, dt, out_dtype):
    g = torch.Generator().manual_seed(m + k)
    a, b = torch.randn(m, k, generator=g).to(DT[dt]).cuda(), (torch.randn(k, n, generator=g) * 1.5 / math.sqrt(k)).to(DT[dt]).cuda()
    bias = torch.randn(n, generator=g).to(out_dtype).cuda()
    got = raw_gemm(a, b, DT[dt], bias=bias, epilogue=epilogue, tuning=(0, 0, 0, split), out_dtype=out_dtype)[0, 0]
    want, magnitude = product(a, b, dt)
    x, u = want + bias.double(), 2.0 ** -24
    # one rounding of the result; the sum's error through a slope of at most 1.13; a handful of fp32 operations on values up to |x| + 1
    bound = UNIT[out_dtype] * ACT[epilogue](x).abs() + 1.13 * (k + 2) * u * (magnitude + bias.double().abs()) + 12 * u * (x.abs() + 1)
    worst = ((got.double() - ACT[epilogue](x)).abs() / bound).max().item()
    assert worst <= 1.0, worst


# one matrix for every batch entry (stride 0) on either side and in either batch dimension, rows on the grid and off it, K split or not
@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("m,n,k", [(130, 200, 64), (65, 131, 300), (64, 64, 2048), (1, 1000, 129)])
@pytest.mark.parametrize("shared", ["a", "b", "a0", "b1", "ab"])
def test_matrices_shared_by_a_batch(m, n, k, shared, split):
    b0, b1 = 3, 2
    g = torch.Generator().manual_seed(m + k)
    na = (1 if shared in ("a", "ab", "a0") else b0, 1 if shared in ("a", "ab") else b1)
    nb = (1 if shared in ("b", "ab") else b0, 1 if shared in ("b", "ab", "b1") else b1)
    a = torch.randn(*na, m, k, generator=g).half().cuda()
    b = (torch.randn(*nb, k, n, generator=g) / math.sqrt(k)).half().cuda()
    strides = [tuple(0 if e == 1 else s for e, s in zip(x.shape[:2], x.stride()[:2])) for x in (a, b)]
    got = raw_gemm(a, b, torch.float16, b0, b1, *strides, tuning=(0, 0, 0, split))
    shape = (b0, b1, m, n)
    close(got, (a.double() @ b.double()).expand(shape), k, (a.double().abs() @ b.double().abs()).expand(shape))


# fp32 results of 16-bit operands: packed, few results, K of 1, a shared matrix
@pytest.mark.parametrize("m,n,k,shared", [(65, 67, 1069, False), (16, 128, 4096, False), (8, 10, 4096, False), (512, 512, 1, False), (130, 200, 2048, True)])
@pytest.mark.parametrize("split", [0, 1])
def test_fp32_results_of_other_products_have_fp32_sums(m, n, k, shared, split):
    g = torch.Generator().manual_seed(k)
    a, b = torch.randn(2 if shared else 1, m, k, generator=g).half().cuda(), (torch.randn(k, n, generator=g) / math.sqrt(k)).half().cuda()
    got = raw_gemm(a, b, torch.float16, 1, 2 if shared else 1, (0, m * k), tuning=(0, 0, 0, split), out_dtype=torch.float32)[0]
    want = a.double() @ b.double()
    # a running fp32 sum of k independent terms errs by about sqrt(k) / 2 roundings of the result's size; the tensor cores by 3e-6 at 4096
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -24 * (1 + math.sqrt(k) / 2)


def test_product_without_scratch():
    """Off the grid with no memory to pack into: the general kernel takes it, and nothing of the refusal stays behind."""
    from metalhlo_b200 import cuda

    g = torch.Generator().manual_seed(11)
    a, b = torch.randn(130, 333, generator=g).half().cuda(), (torch.randn(333, 201, generator=g) / 18).half().cuda()
    bias = torch.randn(201, generator=g).half().cuda()
    want, magnitude = product(a, b, "f16")
    for _ in range(2):
        try:
            assert cuda.lib.mhlo_cuda_debug_refuse_allocs(1) == 0
            close(cuda.gemm(a, b), want, 333, magnitude)
            assert cuda.last_error() == ""
        finally:
            cuda.lib.mhlo_cuda_debug_refuse_allocs(0)
    cuda.lib.mhlo_cuda_debug_refuse_allocs(1)
    try:
        got = cuda.gemm(a, b, bias=bias, epilogue="relu")
    finally:
        cuda.lib.mhlo_cuda_debug_refuse_allocs(0)
    # the product is rounded before the bias there
    assert float((got.double() - torch.relu(want + bias.double())).abs().max()) <= 2 * 2.0 ** -11 * float(want.abs().max() + bias.abs().max())
    close(cuda.gemm(a, b), want, 333, magnitude)


# more batch entries, or more rows, than the general kernel takes: nothing that the other kernels take is handed to it
@pytest.mark.parametrize("dt,out_dtype,b,m,n,k", [(torch.float16, torch.float16, 66000, 64, 65, 17), (torch.float16, torch.float32, 66000, 16, 32, 72),
                                                  (torch.float16, torch.float32, 66000, 40, 45, 41), (torch.float32, torch.float32, 1, 4194304 + 65, 4, 8)])
def test_products_beyond_the_general_kernel(dt, out_dtype, b, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(k)
    x, y = (torch.randn(s, generator=g, device="cuda", dtype=torch.float32).to(dt) for s in ((b, m, k), (b, k, n)))
    got = raw_gemm(x, y, dt, 1, b, (0, m * k), (0, k * n), out_dtype=out_dtype)[0]
    some = slice(0, None, 997) if b > 1 else slice(None)
    rows = slice(None) if b > 1 else slice(0, None, 1009)
    xs, ys = x[some, rows].double(), y[some].double()
    close(got[some, rows], xs @ ys, k, xs.abs() @ ys.abs())


# fp32 results through widened operands: either type, every layout, a matrix shared by a batch, bias and activation
@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("m,n,k", [(300, 257, 65), (33, 61, 600), (1, 3000, 40), (3000, 1, 40)])
@pytest.mark.parametrize("la,lb", [(("row", 0, 0), ("row", 1, 0)), (("row", 0, 1), ("col", 5, 2)), (("col", 3, 0), ("both", 0, 0)), (("both", 0, 0), ("row", 0, 0))])
def test_fp32_results_of_views(m, n, k, la, lb, dt):
    g = torch.Generator().manual_seed(m + k)
    a, b = torch.randn(m, k, generator=g).to(DT[dt]).cuda(), (torch.randn(k, n, generator=g) / math.sqrt(k)).to(DT[dt]).cuda()
    a[0, 0], b[k - 1, n - 1] = 6e-8, -1e-40  # an f16 subnormal and a bf16 one
    views = []
    for x, (order, extra, offset) in ((a, la), (b, lb)):
        inner = x.shape[0] if order == "col" else x.shape[1]
        views.append(strided(x, order, (inner + 7) // 8 * 8 + extra, offset))
    bias = torch.randn(n, generator=g).cuda()
    want, magnitude = product(a, b, dt)
    close(raw_gemm(*views, DT[dt], out_dtype=torch.float32)[0, 0], want, k, magnitude)
    got = raw_gemm(*views, DT[dt], 1, 3, (0, 0), (0, 0), bias=bias, epilogue="relu", out_dtype=torch.float32)[0]
    close(got, torch.relu(want + bias.double()).expand(3, m, n), k + 1, (magnitude + bias.double().abs()).expand(3, m, n))
