"""Calls that take scratch, as the first of a process and inside a stream capture: the graph replays with the buffers' contents."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

COMMON = """
import torch
from metalhlo_b200 import capi, cuda
g = torch.Generator().manual_seed(1)
graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
def replay(x, call, want):
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=stream):
        out = call()
    for _ in range(3):
        x.copy_(torch.randn(x.shape, generator=g))
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        w = want()
        assert float((out.double() - w).abs().max()) <= 2.0 ** -10 * float(w.abs().max()) + 1e-3
    print("replayed")
"""

PACKED = COMMON + """
a, b = torch.randn(130, 333, generator=g).half().cuda(), torch.randn(333, 201, generator=g).half().cuda()
out = torch.zeros(130, 201, dtype=torch.float16, device="cuda")
replay(a, lambda: cuda.gemm(a, b, out=out), lambda: a.double() @ b.double())
"""

REDUCED = COMMON + """
n = 1 << 20
text = f"func.func @main(%x: tensor<{n}xf32>) -> tensor<f32> {{\\n  %z = stablehlo.constant dense<0.0> : tensor<f32>\\n  %0 = stablehlo.reduce(%x init: %z) " \
       f"applies stablehlo.add across dimensions = [0] : (tensor<{n}xf32>, tensor<f32>) -> tensor<f32>\\n  return %0 : tensor<f32>\\n}}\\n"
exe = capi.Client().compile(text, opt_level=3)
x, out = torch.randn(n, generator=g).cuda(), torch.zeros((), device="cuda")
def call():
    exe.execute_on_device([x.data_ptr()], [out.data_ptr()], torch.cuda.current_stream().cuda_stream)
    return out
replay(x, call, lambda: x.double().sum())
"""


@pytest.mark.parametrize("program", [PACKED, REDUCED], ids=["packed product", "split reduction"])
def test_first_scratch_of_a_process_under_capture(program):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", program], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "replayed" in r.stdout, r.stderr[-2000:]


def test_scratch_of_destroyed_graphs_goes_back_when_memory_runs_short():
    import ctypes as C
    import gc

    import torch

    from metalhlo_b200 import cuda

    a, b = torch.zeros(8192, 20001, dtype=torch.float16, device="cuda"), torch.zeros(20001, 8191, dtype=torch.float16, device="cuda")
    out = torch.empty(8192, 8191, dtype=torch.float16, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    before = torch.cuda.mem_get_info()[0]
    with torch.cuda.graph(graph, stream=stream):
        cuda.gemm(a, b, out=out)  # about 650 MB of packed operands, owned by the graph
    graph.replay()
    torch.cuda.synchronize()
    del graph
    gc.collect()
    p = C.c_void_p()
    assert cuda.lib.mhlo_cuda_alloc(1 << 50, C.byref(p)) == 6 and not p.value  # more than there is
    assert torch.cuda.mem_get_info()[0] >= before - (64 << 20)
    small = torch.zeros(4, device="cuda")
    cuda.check(cuda.lib.mhlo_cuda_memset(small.data_ptr(), 1, 16, torch.cuda.current_stream().cuda_stream))  # nothing of the refusal is left
    torch.cuda.synchronize()
