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
