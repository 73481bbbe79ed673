"""Several row operations of one input in one launch: what joins a group, and results equal to the single kernels'."""
import ctypes as C

import pytest
import torch

from metalhlo_b200 import capi, modules
from metalhlo_b200.modules import layer_norm_text, softmax_text, tt


def program(rows, hidden, dt, scale="4.000000e+00", second_use=False, late_gamma=False):
    """LayerNorm(x), RMSNorm(x) with gamma and softmax(x * scale); the RMSNorm's gamma made from the LayerNorm's result if late."""
    t, tv = tt((rows, hidden), dt), tt((hidden,), dt)
    body, ln = layer_norm_text("%arg0", (rows, hidden), dt, "%arg1", "%arg2", prefix="a")
    gamma = "%arg1"
    if late_gamma:
        body += (f"    %row = stablehlo.slice {ln} [0:1, 0:{hidden}] : ({t}) -> {tt((1, hidden), dt)}\n"
                 f"    %late = stablehlo.reshape %row : ({tt((1, hidden), dt)}) -> {tv}\n")
        gamma = "%late"
    text, rms = layer_norm_text("%arg0", (rows, hidden), dt, gamma, None, rms=True, prefix="b")
    body += text + f"    %c = stablehlo.constant dense<{scale}> : {t}\n    %xs = stablehlo.multiply %arg0, %c : {t}\n"
    text, sm = softmax_text("%xs", (rows, hidden), dt, 1, prefix="c")
    outs = [ln, rms, sm] + (["%xs"] if second_use else [])
    return modules.func([t, tv, tv], [t] * len(outs), (body + text).rstrip("\n"), ", ".join(outs))


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
def test_what_joins_a_group(dt):
    assert capi.plan_text(program(6, 64, dt), 3)[0] == ["fused_row_group(x3)"]
    # a scaled input that something else reads is computed, and the softmax reads that
    steps = capi.plan_text(program(6, 64, dt, second_use=True), 3)[0]
    assert "fused_row_group(x2)" in steps and "fused_softmax" in steps
    steps = capi.plan_text(program(6, 64, dt, late_gamma=True), 3)[0]
    assert "fused_rms_norm" in steps or "fused_row_group(x2)" in steps
    assert "fused_row_group(x3)" not in steps
    # rows that are no whole number of 16-byte vectors, and rows too long for the registers
    for hidden in (63, 16384 + 64):
        assert not any("row_group" in s for s in capi.plan_text(program(2, hidden, dt), 3)[0])
    steps = capi.plan_text(program(6, 64, dt, scale="0.000000e+00"), 3)[0]
    assert "fused_row_group(x3)" not in steps


TORCH = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def row_group(x, heads):
    from metalhlo_b200 import cuda

    outs = [torch.empty_like(x) for _ in heads]
    return row_group_into(x, heads, outs)


def row_group_into(x, heads, outs):
    from metalhlo_b200 import cuda

    code = {torch.float32: capi.F32, torch.float16: capi.F16, torch.bfloat16: capi.BF16}[x.dtype]
    group = cuda.RowHeads(count=len(heads))
    for k, (op, gamma, beta, value) in enumerate(heads):
        group.head[k] = cuda.RowHead(None if gamma is None else gamma.data_ptr(), None if beta is None else beta.data_ptr(), outs[k].data_ptr(), value, op)
    assert cuda.lib.mhlo_cuda_row_group(code, x.data_ptr(), C.byref(group), x.shape[0], x.shape[1], torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return outs


def singles(x, heads):
    from metalhlo_b200 import cuda

    out = []
    for op, gamma, beta, value in heads:
        if op == 0:
            out.append(cuda.layer_norm(x, gamma, beta, eps=value))
        elif op == 1:
            out.append(cuda.rms_norm(x, gamma, eps=value))
        else:
            out.append(cuda.softmax(x * torch.tensor(value, dtype=x.dtype, device="cuda")))
    return out


def same_bits(got, want):
    # every value, NaNs at the same places
    return torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.nan_to_num(got), torch.nan_to_num(want))


# one warp and several, rows that leave threads idle, 1 to 8 vectors a thread, fewer and more rows than the grid
@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("rows,hidden", [(1, 8), (5, 40), (7, 256), (3, 768), (1999, 1024), (33, 1032), (9, 4096), (4, 4104), (3, 8192), (2, 12288), (2, 16384)])
def test_group_matches_single_kernels(rows, hidden, dt):
    g = torch.Generator().manual_seed(rows + hidden)
    x = torch.randn(rows, hidden, generator=g)
    x[0, 1], x[rows // 2, 2], x[-1] = float("inf"), -1e4, 2.0
    x = x.to(TORCH[dt]).cuda()
    gamma, beta, gamma2 = ((torch.randn(hidden, generator=g) * 0.1 + 1).to(TORCH[dt]).cuda() for _ in range(3))
    third = float(torch.tensor(0.3, dtype=TORCH[dt]))
    for heads in ([(0, gamma, beta, 1e-5), (1, gamma, None, 1e-6), (2, None, None, 4.0)], [(2, None, None, -0.5), (0, gamma2, None, 1e-5)],
                  [(0, gamma, beta, 1e-5), (0, gamma2, beta, 1e-3)], [(1, None, None, 1e-5), (2, None, None, 1.0)], [(2, None, None, third)]):
        for got, want in zip(row_group(x, heads), singles(x, heads)):
            assert same_bits(got, want), heads


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,offset", [(512, 1), (101, 0)])
def test_group_off_the_16_byte_grid(hidden, offset):
    g = torch.Generator().manual_seed(hidden)
    rows = 6
    x = torch.randn(rows * hidden + offset, generator=g).to(torch.bfloat16).cuda()[offset:].view(rows, hidden)
    gamma = torch.ones(hidden, dtype=torch.bfloat16, device="cuda")
    heads = [(0, gamma, gamma, 1e-5), (1, gamma, None, 1e-5), (2, None, None, 3.0)]
    for got, want in zip(row_group(x, heads), singles(x, heads)):
        # the strided kernel sums in another order: one rounding of the result, 2^-8 of it, and 1e-6 of the sums
        assert torch.allclose(got.float(), want.float(), rtol=2.0 ** -7, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["bf16", "f32"])
@pytest.mark.parametrize("rows,hidden", [(3, 64), (300, 4096)])
def test_group_in_a_program(rows, hidden, dt):
    from parity import assert_close
    import oracle

    g = torch.Generator().manual_seed(5)
    x, gamma, beta = torch.randn(rows, hidden, generator=g), 1 + 0.1 * torch.randn(hidden, generator=g), 0.1 * torch.randn(hidden, generator=g)
    x, gamma, beta = (t.to(TORCH[dt]) for t in (x, gamma, beta))
    client = capi.Client()
    exe = client.compile(program(rows, hidden, dt), opt_level=3)
    assert "fused_row_group(x3)" in exe.steps
    outs = [o.to_numpy().astype("float64") for o in exe.execute([client.buffer(t) for t in (x, gamma, beta)])]
    tol = 2e-2 if dt == "bf16" else 1e-5
    for got, want in zip(outs, (oracle.layer_norm(x, gamma, beta), oracle.rms_norm(x, gamma), oracle.softmax(x * 4))):
        assert_close(got, want, tol, f"group {dt}")


@pytest.mark.gpu
@pytest.mark.parametrize("rows,hidden,offset", [(300, 1024, 0), (3, 40, 0), (2000, 4096, 0), (6, 512, 1), (5, 101, 0)])
@pytest.mark.parametrize("place", [0, 1, 2])
def test_one_result_may_take_the_place_of_x(rows, hidden, offset, place):
    g = torch.Generator().manual_seed(hidden + place)
    flat = torch.randn(rows * hidden + offset, generator=g).to(torch.bfloat16).cuda()
    x = flat[offset:].view(rows, hidden)
    gamma = (torch.randn(hidden, generator=g) * 0.1 + 1).to(torch.bfloat16).cuda()
    heads = [(0, gamma, gamma, 1e-5), (1, gamma, None, 1e-6), (2, None, None, 3.0)]
    want = row_group(x.clone() if not offset else flat.clone()[offset:].view(rows, hidden), heads)
    outs = [torch.empty_like(flat)[offset:].view(rows, hidden) for _ in heads]
    outs[place] = x
    for got, w in zip(row_group_into(x, heads, outs), want):
        assert same_bits(got, w)


def program_with_a_step_between(hidden, dt, returned):
    """LayerNorm(x), LayerNorm(x) + w, RMSNorm(x): the RMSNorm returned, or only read by a sum."""
    t, tv = tt((4, hidden), dt), tt((hidden,), dt)
    body, ln = layer_norm_text("%arg0", (4, hidden), dt, "%arg1", "%arg1", prefix="a")
    body += f"    %w2 = stablehlo.add {ln}, %arg2 : {t}\n"
    text, rms = layer_norm_text("%arg0", (4, hidden), dt, "%arg1", None, rms=True, prefix="b")
    body += text
    if not returned:
        body, rms = body + f"    %last = stablehlo.add {rms}, {rms} : {t}\n", "%last"
    return modules.func([t, tv, t], [t] * 2, body.rstrip("\n"), f"%w2, {rms}")


def test_a_returned_result_does_not_move_across_other_steps():
    steps = capi.plan_text(program_with_a_step_between(64, "f32", True), 3)[0]
    assert "fused_layer_norm" in steps and "fused_rms_norm" in steps
    assert "fused_row_group(x2)" in capi.plan_text(program_with_a_step_between(64, "f32", False), 3)[0]


@pytest.mark.gpu
def test_a_result_bound_to_an_argument_that_a_step_between_reads():
    exe = capi.Client().compile(program_with_a_step_between(64, "f32", True), opt_level=3)
    g = torch.Generator().manual_seed(3)
    x, gamma, w = (torch.randn(4, 64, generator=g).cuda(), torch.randn(64, generator=g).cuda(), torch.randn(4, 64, generator=g).cuda())
    torch.cuda.synchronize()
    plain, bound = [torch.empty_like(x) for _ in range(2)], [torch.empty_like(x)]
    stream = torch.cuda.current_stream().cuda_stream
    exe.execute_on_device([t.data_ptr() for t in (x, gamma, w)], [t.data_ptr() for t in plain], stream)
    mine = w.clone()
    exe.execute_on_device([t.data_ptr() for t in (x, gamma, mine)], [t.data_ptr() for t in bound + [mine]], stream)
    torch.cuda.synchronize()
    for got, want in zip(bound + [mine], plain):
        assert torch.equal(got, want)
