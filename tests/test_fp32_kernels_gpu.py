"""fp32 products and attention on the FMA units at the edges of their tiles and of their dispatch."""
import math

import numpy as np
import pytest
import torch

import oracle
from parity import assert_close, to_np

pytestmark = pytest.mark.gpu


def cuda_mod():
    from metalhlo_b200 import cuda

    return cuda


# 16 x 64, 64 x 64 and 128 x 128 tiles (the last from 236 tiles on), K split over clusters, panels of 16 / 32 / 64 steps;
# extents off the 16-byte grid take the 4-byte copies
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (1, 1000, 777), (16, 64, 64), (17, 65, 33), (64, 64, 32), (65, 129, 31), (128, 128, 2048), (100, 36, 1029),
                                   (2048, 2048, 48), (2050, 2051, 17)])
def test_gemm_fp32(trans_a, trans_b, m, n, k):
    g = torch.Generator().manual_seed(m + n + k)
    a = torch.randn((k, m) if trans_a else (m, k), generator=g)
    b = torch.randn((n, k) if trans_b else (k, n), generator=g)
    bias = torch.randn(n, generator=g)
    got = cuda_mod().gemm(a.cuda(), b.cuda(), bias=bias.cuda(), trans_a=trans_a, trans_b=trans_b).double().cpu()
    da, db = (a.double().T if trans_a else a.double()), (b.double().T if trans_b else b.double())
    want = da @ db + bias.double()
    # any order of k + 1 fp32 additions of fp32 products: |error| <= (k + 2) u sum |terms|, u = 2^-24
    bound = (k + 2) * 2.0 ** -24 * (da.abs() @ db.abs() + bias.double().abs())
    assert bool(((got - want).abs() <= bound).all())


@pytest.mark.parametrize("batch", [(5,), (2, 3)])
@pytest.mark.parametrize("epilogue", ["none", "gelu_tanh", "relu"])
def test_gemm_fp32_batched_with_epilogue(batch, epilogue):
    m, n, k = 70, 132, 130
    g = torch.Generator().manual_seed(1)
    a, b = torch.randn(*batch, m, k, generator=g) / math.sqrt(k), torch.randn(*batch, k, n, generator=g)
    bias = torch.randn(n, generator=g)
    got = cuda_mod().gemm(a.cuda(), b.cuda(), bias=bias.cuda(), epilogue=epilogue)
    want = a.double() @ b.double() + bias.double()
    want = {"none": lambda x: x, "relu": torch.relu, "gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}[epilogue](want)
    assert_close(to_np(got), want.numpy(), 1e-5, f"gemm fp32 {batch} {epilogue}")


# row groups of 32, 64 and 128; one or two warps per group (head dimensions up to 64 and up to 128); keys shared by a cluster
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,h,sq,sk,d", [(1, 1, 1, 1, 64), (1, 2, 33, 65, 64), (1, 1, 300, 1030, 64), (2, 40, 130, 96, 40), (3, 50, 129, 257, 64),
                                         (1, 3, 31, 33, 128), (2, 5, 97, 300, 80), (3, 50, 128, 129, 128), (1, 2, 65, 64, 33)])
def test_attention_fp32(causal, b, h, sq, sk, d):
    g = torch.Generator().manual_seed(sq + sk + d)
    q, k, v = (torch.randn(b, h, s, d, generator=g) for s in (sq, sk, sk))
    scale = 1 / math.sqrt(d)
    got = cuda_mod().attention(q.cuda(), k.cuda(), v.cuda(), scale, causal=causal)
    assert_close(to_np(got), oracle.attention(q, k, v, scale, causal=causal), 1e-5, f"{sq}x{sk} d{d}",
                 magnitude=oracle.attention(q, k, v.abs(), scale, causal=causal))


@pytest.mark.parametrize("d", [64, 100])
def test_attention_fp32_mask_and_interleaved_heads(d):
    g = torch.Generator().manual_seed(d)
    q, k, v = (torch.randn(2, s, 3, d, generator=g) for s in (70, 90, 90))
    mask = torch.randn(70, 90, generator=g)
    mask[3] = -math.inf  # a row that sees nothing
    mask[5, 1:] = -math.inf
    got = to_np(cuda_mod().attention(q.cuda(), k.cuda(), v.cuda(), 0.1, mask=mask.cuda(), layout="BSHD")).transpose(0, 2, 1, 3)
    qt, kt, vt = (t.permute(0, 2, 1, 3).contiguous() for t in (q, k, v))
    s = qt.double() @ kt.double().transpose(-1, -2) * 0.1 + mask.double()
    p = torch.nan_to_num(torch.softmax(s, -1), nan=0.0)
    assert np.all(got[:, :, 3] == 0)
    assert_close(got, (p @ vt.double()).numpy(), 1e-5, "masked", magnitude=(p @ vt.double().abs()).numpy())


# the fp32 kernel with and without its keys shared by a cluster, one and two warps per row group; f16 rows of 33 take the general kernel
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dt,b,h,sq,sk,d", [(torch.float32, 1, 1, 300, 1030, 64), (torch.float32, 2, 40, 130, 96, 40), (torch.float32, 3, 50, 129, 257, 64),
                                            (torch.float32, 1, 3, 31, 33, 128), (torch.float32, 3, 50, 128, 129, 128), (torch.float16, 1, 2, 50, 70, 33)])
def test_attention_hands_nans_on(causal, dt, b, h, sq, sk, d):
    g = torch.Generator().manual_seed(sq + d)
    q, k, v = (torch.randn(b, h, s, d, generator=g).to(dt) for s in (sq, sk, sk))
    scale = 1 / math.sqrt(d)
    clean = cuda_mod().attention(q.cuda(), k.cuda(), v.cuda(), scale, causal=causal).cpu()
    bad = q.clone()
    bad[0, 0, 7, 0] = math.nan  # every score of one row
    got = cuda_mod().attention(bad.cuda(), k.cuda(), v.cuda(), scale, causal=causal).cpu()
    assert bool(torch.isnan(got[0, 0, 7]).all())
    got[0, 0, 7] = clean[0, 0, 7]
    assert torch.equal(got, clean)
    bad = k.clone()
    bad[0, 0, :64] = math.nan  # every key of the first blocks: all rows see key 0
    got = cuda_mod().attention(q.cuda(), bad.cuda(), v.cuda(), scale, causal=causal).cpu()
    assert bool(torch.isnan(got[0, 0]).all()) and torch.equal(got.flatten(0, 1)[1:], clean.flatten(0, 1)[1:])


# rows of several warps and CTAs, keys shared by a cluster, two warps per row group, more keys than queries and fewer
@pytest.mark.parametrize("b,h,sq,sk,d", [(1, 1, 300, 300, 64), (1, 1, 300, 1030, 64), (3, 50, 129, 257, 64), (2, 40, 130, 96, 40), (1, 3, 190, 190, 128),
                                         (3, 50, 128, 129, 100)])
def test_attention_rows_do_not_touch_values_behind_the_causal_limit(b, h, sq, sk, d):
    g = torch.Generator().manual_seed(sq + d)
    q, k, v = (torch.randn(b, h, s, d, generator=g) for s in (sq, sk, sk))
    scale = 1 / math.sqrt(d)
    want = oracle.attention(q, k, v, scale, causal=True)
    magnitude = oracle.attention(q, k, v.abs(), scale, causal=True)
    for limit in (1, 37, 64, min(sq, sk) - 1):
        for bad in (math.inf, math.nan):
            k2, v2 = k.clone(), v.clone()
            k2[:, :, limit:], v2[:, :, limit:] = bad, bad
            got = to_np(cuda_mod().attention(q.cuda(), k2.cuda(), v2.cuda(), scale, causal=True))
            assert_close(got[:, :, :limit], want[:, :, :limit], 1e-5, f"{limit} {bad}", magnitude=magnitude[:, :, :limit])
            assert np.isnan(got[:, :, limit:]).all()


def test_gemm_fp32_empty_and_refused_extents():
    import ctypes as C

    cuda = cuda_mod()
    bias = torch.zeros(6).cuda()
    for shape_a, shape_b in (((0, 4, 5), (0, 5, 6)), ((2, 0, 4, 5), (2, 0, 5, 6)), ((3, 0, 5), (3, 5, 6))):
        got = cuda.gemm(torch.zeros(shape_a).cuda(), torch.zeros(shape_b).cuda(), bias=bias, epilogue="relu")
        assert got.shape == (*shape_a[:-1], 6) and got.numel() == 0
    x = torch.ones(64).cuda()
    for b0, b1, m, n, k in ((-1, -1, 4, 4, 4), (1, 1, -4, -4, 4), (1, 1, 4, 4, -4)):
        status = cuda.lib.mhlo_cuda_gemm(cuda.F32, cuda.F32, x.data_ptr(), cuda._i64s([0, 0, 4, 1]), x.data_ptr(), cuda._i64s([0, 0, 4, 1]),
                                         x.data_ptr(), b0, b1, m, n, k, None, 0, None)
        assert status == 10, (b0, b1, m, n, k)
    torch.cuda.synchronize()
    assert bool((x == 1).all())



# either side of the lines of the dispatch: K of 16 and 17 with 296 tiles and more; 128 x 128 tiles filled to 0.6 or not, K of 64 and 65
@pytest.mark.parametrize("b,m,n,k", [(296, 16, 64, 16), (297, 16, 64, 16), (297, 1, 3, 4), (297, 16, 64, 17), (296, 17, 64, 16), (297, 17, 64, 16), (297, 64, 33, 17),
                                     (1, 19000, 5, 16), (1, 30208, 77, 65), (1, 30208, 76, 65), (1, 77, 30208, 65), (1, 30208, 128, 64), (60, 129, 200, 70),
                                     (1, 40000, 1, 100)])
def test_gemm_fp32_lines_of_the_dispatch(b, m, n, k):
    g = torch.Generator().manual_seed(b + m + n + k)
    x, y = torch.randn(b, m, k, generator=g), torch.randn(b, k, n, generator=g)
    got = cuda_mod().gemm(x.cuda(), y.cuda()).double().cpu()
    bound = (k + 2) * 2.0 ** -24 * (x.double().abs() @ y.double().abs())
    assert bool(((got - x.double() @ y.double()).abs() <= bound).all())


# shapes either side of the choice between tiles and a warp per query row: a decoding step of few and of many heads, few keys, few queries
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,h,sq,sk,d", [(1, 1, 1, 300, 64), (40, 50, 1, 100, 64), (40, 50, 3, 100, 64), (40, 50, 8, 100, 64), (1, 1, 32, 8, 64), (1, 1, 32, 40, 64),
                                         (30, 10, 1, 200, 128), (30, 10, 9, 200, 128), (2, 2, 5, 64, 4), (2, 2, 5, 300, 4), (3, 1, 700, 3, 20)])
def test_attention_fp32_few_rows_or_keys(causal, b, h, sq, sk, d):
    g = torch.Generator().manual_seed(sq + sk + d)
    q, k, v = (torch.randn(b, h, s, d, generator=g) for s in (sq, sk, sk))
    scale = 1 / math.sqrt(d)
    s = q.double() @ k.double().transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(sq, sk, dtype=torch.bool).triu(1), -math.inf)
    p = torch.softmax(s, -1)
    got = cuda_mod().attention(q.cuda(), k.cuda(), v.cuda(), scale, causal=causal)
    assert_close(to_np(got), (p @ v.double()).numpy(), 1e-5, f"{sq}x{sk} d{d}", magnitude=(p @ v.double().abs()).numpy())
