"""Products whose sum over K is split over a cluster: widths of 64 and 128 columns, clusters of 2, 4 and 8, CTAs without a share of K."""
import math

import pytest
import torch

from test_gemm_layouts_gpu import ACT, DT, UNIT, close, product, raw_gemm, strided

pytestmark = pytest.mark.gpu

SPLIT = (0, 0, 0, 1)

# (m, n, k) and what the choice by costs makes of them
SHAPES = [(128, 64, 576),     # 64 columns, cluster of 8: nine steps in shares of two, three CTAs without any
          (33, 61, 1537),     # the same, ragged in every extent (N odd: results stored one by one)
          (201, 768, 768),    # 64 columns, cluster of 4
          (201, 2304, 768),   # 64 columns, cluster of 2
          (1024, 768, 3072),  # 128 columns, cluster of 2
          (300, 1540, 8200),  # 128 columns, cluster of 4
          (300, 1002, 16392)]  # 128 columns, cluster of 8


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("la,lb", [("row", "row"), ("col", "row"), ("row", "col"), ("col", "col")])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_majors(m, n, k, la, lb, dt):
    g = torch.Generator().manual_seed(m + n)
    a, b = torch.randn(m, k, generator=g).to(DT[dt]).cuda(), (torch.randn(k, n, generator=g) / math.sqrt(k)).to(DT[dt]).cuda()
    views = [strided(x, order, ((x.shape[0] if order == "col" else x.shape[1]) + 7) // 8 * 8) for x, order in ((a, la), (b, lb))]
    want, magnitude = product(a, b, dt)
    got = raw_gemm(*views, DT[dt], tuning=SPLIT)[0, 0]
    close(got, want, k, magnitude)
    assert torch.equal(got, raw_gemm(*views, DT[dt], tuning=SPLIT)[0, 0])  # the same sum on every run


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_results_bias_and_activations(m, n, k, out_dtype):
    g = torch.Generator().manual_seed(m + k)
    pad = (n + 7) // 8 * 8
    a = strided(torch.randn(m, k, generator=g).bfloat16().cuda(), "row", (k + 7) // 8 * 8)
    b = strided((torch.randn(k, n, generator=g) * 1.5 / math.sqrt(k)).bfloat16().cuda(), "row", pad)
    bias = torch.randn(n, generator=g).to(out_dtype).cuda()
    want, magnitude = product(a, b, "bf16")
    x, u = want + bias.double(), 2.0 ** -24
    for epilogue in sorted(ACT):
        got = raw_gemm(a, b, torch.bfloat16, bias=bias, epilogue=epilogue, tuning=SPLIT, out_dtype=out_dtype)[0, 0]
        # as for the other products; the hardware's tanh and exponential are good to 2^-10 of the result's scale
        approximate = 2.0 ** -10 * (x.abs() + 1) if m * n >= 64 * 64 and epilogue in ("gelu_tanh", "silu", "sigmoid") else 0.0
        bound = UNIT[out_dtype] * ACT[epilogue](x).abs() + 1.13 * (k + 2) * u * (magnitude + bias.double().abs()) + 12 * u * (x.abs() + 1) + approximate
        worst = ((got.double() - ACT[epilogue](x)).abs() / bound).max().item()
        assert worst <= 1.0, (epilogue, worst)


@pytest.mark.parametrize("b0,b1,m,n,k", [(3, 2, 100, 64, 576), (1, 5, 128, 100, 2048), (4, 1, 1, 256, 8192)])
def test_batches(b0, b1, m, n, k):
    g = torch.Generator().manual_seed(n)
    a, b = torch.randn(b0, b1, m, k, generator=g).half().cuda(), torch.zeros(b0, b1, k, (n + 7) // 8 * 8).half().cuda()
    b[..., :n] = (torch.randn(b0, b1, k, n, generator=g) / math.sqrt(k)).half().cuda()
    b = b[..., :n]
    got = raw_gemm(a, b, torch.float16, b0, b1, a.stride()[:2], b.stride()[:2], tuning=SPLIT)
    close(got, a.double() @ b.double(), k, a.double().abs() @ b.double().abs())
