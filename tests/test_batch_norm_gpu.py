"""Batch norm with the channels last: channels that fill vectors and that do not, fewer and more rows than threads, off the 16-byte grid."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,unit", [(torch.float32, 2.0 ** -24), (torch.float16, 2.0 ** -11), (torch.bfloat16, 2.0 ** -8)])
@pytest.mark.parametrize("rows,channels,offset", [(1, 1, 0), (5, 8, 0), (300, 7, 0), (4099, 24, 0), (70000, 64, 0), (3, 4104, 0), (2, 300001, 0), (37, 64, 1)])
def test_batch_norm(rows, channels, offset, dt, unit):
    from metalhlo_b200 import capi, cuda

    g = torch.Generator().manual_seed(rows + channels)
    x = torch.randn(rows * channels + offset, generator=g).to(dt).cuda()[offset:].view(rows, channels)
    scale, shift, mean = (torch.randn(channels, generator=g).to(dt).cuda() for _ in range(3))
    variance = (torch.rand(channels, generator=g) + 0.5).to(dt).cuda()
    y = torch.empty_like(x)
    code = {torch.float32: capi.F32, torch.float16: capi.F16, torch.bfloat16: capi.BF16}[dt]
    assert cuda.lib.mhlo_cuda_batch_norm(code, x.data_ptr(), scale.data_ptr(), shift.data_ptr(), mean.data_ptr(), variance.data_ptr(), y.data_ptr(),
                                         rows, channels, 1e-3, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    d, s = (x.double() - mean.double()) * scale.double() / torch.sqrt(variance.double() + 1e-3), shift.double()
    # seven fp32 operations on the product, one on the sum, one rounding of the result (and of f16's subnormals)
    assert bool(((y.double() - (d + s)).abs() <= 8 * 2.0 ** -24 * (d.abs() + s.abs()) + unit * (d + s).abs() + 2.0 ** -24).all())
