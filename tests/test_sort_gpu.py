"""Sorts at the edges of the radix tiles (512 to 8192 keys) and of the chunked path behind them; keys of up to 32 bits and their payloads."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FROM = {torch.float32: "F32", torch.float16: "F16", torch.bfloat16: "BF16", torch.int32: "I32", torch.int16: "I16", torch.int8: "I8", torch.uint8: "UI8",
        torch.int64: "I64", torch.float64: "F64"}


def sort(operands, dimension, flags):
    from metalhlo_b200 import capi, cuda

    shape = (C.c_int64 * operands[0].dim())(*operands[0].shape)
    outs = [torch.empty_like(t) for t in operands]
    need = cuda.lib.mhlo_cuda_sort_scratch_bytes(shape, len(shape), dimension)
    scratch = torch.empty(max(1, need), dtype=torch.uint8, device="cuda")
    n = len(operands)
    pointers, results = (C.c_void_p * n)(*(t.data_ptr() for t in operands)), (C.c_void_p * n)(*(t.data_ptr() for t in outs))
    codes = (C.c_int32 * n)(*(getattr(capi, FROM[t.dtype]) for t in operands))
    assert cuda.lib.mhlo_cuda_sort(pointers, results, codes, n, shape, len(shape), dimension, flags, scratch.data_ptr(), need,
                                   torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return outs


def order(keys, dimension, flags):
    """Stable permutation along `dimension`: the total order of the bits, -0 = +0 with bit 1 of the flags."""
    k = keys.float().numpy() if keys.dtype in (torch.bfloat16, torch.float16) else keys.numpy()
    if k.dtype == np.float32:
        b = k.view(np.int32).astype(np.int64)
        k = np.where(b < 0, -(b & 0x7fffffff) - 1, b)
        if flags & 2:
            k = np.where(k == -1, 0, k)
    k = k.astype(np.int64)
    return np.argsort(-k if flags & 1 else k, axis=dimension, kind="stable")


def draw(n, dt, g, rows=3):
    if dt.is_floating_point:
        x = torch.randn(rows, n, generator=g)
        x[:, ::7] = torch.round(x[:, ::7])  # ties, and zeros of both signs
        x[0, 1::11], x[0, 2::13], x[0, 3::17] = float("inf"), float("-inf"), float("nan")
        x[-1] = 1.5  # every key the same
        return x.to(dt)
    info = torch.iinfo(dt)
    x = torch.randint(info.min, info.max, (rows, n), generator=g, dtype=torch.int64)
    x[0, ::5], x[0, 1::5] = info.max, info.min  # the largest key is the padding's as well
    return x.to(dt)


def check(keys, dimension, flags, payloads=()):
    places = torch.arange(keys.shape[dimension], dtype=torch.int32)
    places = (places if dimension == keys.dim() - 1 else places[:, None]).expand(keys.shape).contiguous()
    operands = [keys, places, *payloads]
    outs = sort([t.cuda() for t in operands], dimension, flags)
    p = torch.from_numpy(order(keys, dimension, flags))
    bits = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}
    for got, t in zip(outs, operands):
        as_bits = bits[t.element_size()]
        assert torch.equal(got.cpu().view(as_bits), torch.gather(t.view(as_bits), dimension, p))


@pytest.mark.parametrize("flags", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 63, 127, 128, 129, 255, 256, 257, 480, 511, 512, 513, 1023, 1025, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 16384, 16385, 40000])
def test_sort_lengths(n, flags):
    check(draw(n, torch.float32, torch.Generator().manual_seed(n + flags)), 1, flags)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.int32, torch.int16, torch.int8, torch.uint8])
@pytest.mark.parametrize("n", [300, 1500, 5000, 9000])
def test_sort_key_types_with_payloads_of_every_width(dt, n):
    g = torch.Generator().manual_seed(n)
    payloads = [draw(n, t, g) for t in (torch.int8, torch.int16, torch.float32, torch.int64)]
    for flags in (0, 1):
        check(draw(n, dt, g), 1, flags, payloads)


@pytest.mark.parametrize("n", [200, 3000, 10000])
def test_sort_along_the_first_dimension(n):
    g = torch.Generator().manual_seed(n)
    check(draw(n, torch.float32, g, rows=5).T.contiguous(), 0, 0, [draw(n, torch.int16, g, rows=5).T.contiguous()])


# short slices take the radix passes only when there are many: one warp and more, remainders, and more slices than the grid
@pytest.mark.parametrize("rows,n", [(148 * 32 + 5, 129), (148 * 32 + 5, 260), (2400, 480), (2400, 512), (1300, 513), (1300, 1023), (700, 1025), (400, 2048)])
def test_sort_many_short_slices(rows, n):
    check(draw(n, torch.float32, torch.Generator().manual_seed(n), rows=rows), 1, 0)
