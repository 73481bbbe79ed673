"""mhlo_cuda_elementwise called directly: operands that name one register several times."""
import ctypes as C
import itertools
import os
import re

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def opcodes():
    with open(os.path.join(ROOT, "include", "mhlo_cuda.h")) as f:
        body = re.search(r"MHLO_EW_COPY = 0.*?MHLO_EW_OP_COUNT", f.read(), re.S).group(0)
    names = re.findall(r"MHLO_EW_\w+", re.sub(r"/\*.*?\*/", "", body, flags=re.S))
    return {n[len("MHLO_EW_"):]: i for i, n in enumerate(names)}


OP = opcodes()


def run(inputs, prog, out):
    from metalhlo_b200 import cuda

    views = (cuda.View * max(len(inputs), 1))()
    for v, t in zip(views, inputs):
        v.base, v.dtype, v.rank = t.data_ptr(), cuda.torch_dtype_code(t.dtype), t.dim()
        for d in range(t.dim()):
            v.shape[d], v.stride[d] = t.shape[d], t.stride(d)
    insts = (cuda.EwInst * len(prog))(*[cuda.EwInst(op, a, b, c, imm) for op, a, b, c, imm in prog])
    cuda.check(cuda.lib.mhlo_cuda_elementwise(views, len(inputs), insts, len(prog), out.data_ptr(), cuda.torch_dtype_code(out.dtype),
                                              cuda._i64s(out.shape), out.dim(), torch.cuda.current_stream().cuda_stream))


def test_opcodes_are_read_from_the_header():
    assert (OP["COPY"], OP["IMM"], OP["ADD"]) == (0, 1, 3) and OP["CLAMP"] == OP["SELECT"] + 1


# every assignment of one to three inputs to the three operands, one instruction and the same behind another
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16, torch.float64, torch.int32, torch.int64])
@pytest.mark.parametrize("n_inputs", [1, 2, 3])
def test_operands_may_share_registers(n_inputs, dt):
    g = torch.Generator().manual_seed(n_inputs)
    x = [torch.randint(-2, 3, (37,), generator=g).to(dt).cuda() for _ in range(n_inputs)]
    out = torch.empty_like(x[0])
    for a, b, c in itertools.product(range(n_inputs), repeat=3):
        want = {"SELECT": torch.where(x[a] != 0, x[b], x[c]), "CLAMP": torch.minimum(torch.maximum(x[b], x[a]), x[c]),
                "SUB": x[a] - x[b], "NEG": -x[a]}
        for name, w in want.items():
            run(x, [(OP[name], a, b, c, 0.0)], out)
            assert torch.equal(out, w), (name, a, b, c)
            run(x, [(OP["NEG"], 0, 0, 0, 0.0), (OP[name], a, b, c, 0.0)], out)
            assert torch.equal(out, w), (name, a, b, c, "second instruction")


# one element per thread up to 75776 elements, 4 or 8 beyond; short programs of cheap float operators keep their vectors
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16, torch.float64, torch.int32, torch.int8, torch.int64])
@pytest.mark.parametrize("shape,view", [((1,), None), ((7,), None), ((1001,), "shift"), ((75776,), None), ((75777,), None), ((37, 2049), "columns"),
                                        ((300, 257), "transpose"), ((5, 1, 7, 9), None), ((1000, 3), "row")])
def test_elements_per_thread(shape, view, dt):
    g = torch.Generator().manual_seed(len(shape))
    n = 1
    for e in shape:
        n *= e

    def tensor(k):
        x = torch.randint(-9, 10, (n + 1,), generator=g).to(dt).cuda()
        if view == "shift":
            return x[1:].view(shape)
        if view == "columns":
            return torch.cat([x, x])[:2 * n].view(shape[0], 2 * shape[1])[:, ::2]
        if view == "transpose":
            return x[:n].view(shape[::-1]).t()
        if view == "row" and k == 1:
            return x[:shape[-1]].expand(shape)
        return x[:n].view(shape)

    x, y = tensor(0), tensor(1)
    out = torch.empty(shape, dtype=dt, device="cuda")
    flags = torch.empty(shape, dtype=torch.bool, device="cuda")
    run([x, y], [(OP["SUB"], 0, 1, 0, 0.0)], out)
    assert torch.equal(out, x - y)
    run([x, y], [(OP["CMP_LT"], 0, 1, 0, 0.0)], flags)
    assert torch.equal(flags, x < y)
    # a value kept for the last instruction, one used at once, and a coordinate
    prog = [(OP["MUL"], 0, 1, 0, 0.0), (OP["NEG"], 2, 2, 2, 0.0), (OP["IOTA"], 0, 0, 0, float(len(shape) - 1)), (OP["ADD"], 3, 0, 0, 0.0), (OP["MAX"], 5, 2, 0, 0.0)]
    run([x, y], prog, out)
    prod = (x * y) if dt not in (torch.bfloat16, torch.int8) else (x.to(torch.int32) * y.to(torch.int32)).to(torch.float64)
    want = torch.maximum(-prod + x.to(prod.dtype), prod)
    assert torch.equal(out, want.to(dt) if dt != torch.int8 else want.to(torch.int64).to(torch.int8))


def test_large_programs_from_several_threads():
    """Programs that keep 15, 20 and 22 values (60, 80 and 88 KB of shared memory a CTA), launched by three threads at the same time."""
    import threading

    n, failures = 80000, []

    def kept(count):
        """count results of x * x chained by sums, all of them read again at the end."""
        prog = [(OP["MUL"], 0, 0, 0, 0.0)] + [(OP["ADD"], k, 0, 0, 0.0) for k in range(1, count)]
        total = count
        for k in range(1, 32 - count + 1):
            prog.append((OP["ADD"], total, k, 0, 0.0))
            total = count + k
        return prog

    def expected(x, prog):
        regs = [x]
        for op, a, b, _c, _imm in prog:
            regs.append(regs[a] * regs[b] if op == OP["MUL"] else regs[a] + regs[b])
        return regs[-1]

    def work(count, extra):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                x = torch.full((n,), 0.5, device="cuda")
                y = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
                inputs, prog = [x] + [y] * extra, [(op, a + (extra if a else 0), b + (extra if b else 0), 0, imm) for op, a, b, _c, imm in kept(count)]
                out = torch.empty(n, device="cuda")
                for _ in range(1500):
                    run(inputs, prog, out)
                torch.cuda.current_stream().synchronize()
                assert torch.equal(out, expected(x, kept(count)))
        except Exception as e:  # noqa: BLE001 - reported below, from the main thread
            failures.append(e)

    threads = [threading.Thread(target=work, args=a) for a in ((16, 3), (18, 7), (12, 2))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
