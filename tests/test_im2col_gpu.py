"""Patch matrices of images whose features do not fill 16-byte vectors: every stride, dilation, padding, reversal and group count."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def patches(x, kernel, stride, pad, lhs, rhs, reverse, groups, out_size):
    """[group][batch, out positions][kernel positions, features of the group] of x [batch, spatial.., features], zero outside."""
    batch, features = x.shape[0], x.shape[-1]
    size, per = x.shape[1:-1], features // groups
    rows = []
    for g in range(groups):
        for b in range(batch):
            for od in np.ndindex(*out_size):
                row = []
                for kd in np.ndindex(*kernel):
                    pos = [o * s - p + (k - 1 - t if r else t) * d for o, s, p, t, k, d, r in zip(od, stride, pad, kd, kernel, rhs, reverse)]
                    inside = all(p >= 0 and p % l == 0 and p // l < n for p, l, n in zip(pos, lhs, size))
                    row.append(x[(b, *[p // l for p, l in zip(pos, lhs)])][g * per:(g + 1) * per] if inside else np.zeros(per, x.dtype))
                rows.append(np.concatenate(row))
    return np.stack(rows)


# channels last and first; one, two and three spatial dimensions; taps of 1, 3 and 5 features; rows with and without padding columns
@pytest.mark.parametrize("dt,code", [(np.uint8, "UI8"), (np.uint16, "F16"), (np.uint32, "F32"), (np.uint64, "I64")])
@pytest.mark.parametrize("size,kernel,stride,pad,lhs,rhs,reverse,groups,features", [
    ((9, 8), (3, 3), (2, 2), (0, 1), (1, 1), (1, 1), (0, 0), 1, 3), ((5, 7), (2, 3), (1, 2), (2, 1), (2, 1), (1, 2), (1, 0), 1, 5),
    ((6, 6), (3, 3), (1, 1), (1, 1), (1, 1), (1, 1), (0, 1), 2, 6), ((11,), (4,), (3,), (2,), (1,), (2,), (0,), 1, 3),
    ((4, 3, 5), (2, 2, 2), (1, 1, 2), (1, 0, 1), (1, 2, 1), (1, 1, 1), (0, 1, 0), 3, 3), ((7, 7), (1, 1), (1, 1), (0, 0), (1, 1), (1, 1), (0, 0), 1, 1)])
@pytest.mark.parametrize("channels_first", [False, True])
def test_im2col(dt, code, size, kernel, stride, pad, lhs, rhs, reverse, groups, features, channels_first):
    from metalhlo_b200 import capi, cuda

    rng, batch, ns = np.random.default_rng(features + len(size)), 2, len(size)
    x = rng.integers(1, 200, (batch, *size, features)).astype(dt)
    out_size = tuple(((n - 1) * l + 1 + 2 * p - ((k - 1) * r + 1)) // s + 1 for n, l, p, k, r, s in zip(size, lhs, pad, kernel, rhs, stride))
    want = patches(x, kernel, stride, pad, lhs, rhs, reverse, groups, out_size)
    kept = np.ascontiguousarray(np.moveaxis(x, -1, 1)) if channels_first else x
    strides = [s // kept.itemsize for s in (np.moveaxis(kept, 1, -1) if channels_first else kept).strides]
    conv = cuda.Conv(n_spatial=ns, batch=batch, in_features=features, out_features=groups, feature_group_count=groups, batch_group_count=1,
                     in_batch_stride=strides[0], in_feature_stride=strides[-1])
    for d in range(ns):
        conv.reverse[d], conv.in_size[d], conv.kernel_size[d], conv.out_size[d] = reverse[d], size[d], kernel[d], out_size[d]
        conv.stride[d], conv.pad_low[d], conv.lhs_dilation[d], conv.rhs_dilation[d] = stride[d], pad[d], lhs[d], rhs[d]
        conv.in_spatial_stride[d] = strides[1 + d]
    source = torch.from_numpy(kept.view(np.uint8).reshape(-1).copy()).cuda()
    for pitch in (want.shape[1], -(-want.shape[1] // 16) * 16, -(-want.shape[1] // 16) * 16 + 8):
        cols = torch.full((want.shape[0] * pitch * x.itemsize,), 255, dtype=torch.uint8, device="cuda")
        assert cuda.lib.mhlo_cuda_im2col(getattr(capi, code), source.data_ptr(), cols.data_ptr(), pitch, C.byref(conv),
                                         torch.cuda.current_stream().cuda_stream) == 0
        got = cols.cpu().numpy().view(dt).reshape(want.shape[0], pitch)
        assert np.array_equal(got[:, :want.shape[1]], want) and not got[:, want.shape[1]:].any()
