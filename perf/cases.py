"""The work that is timed: what a program that uses this backend has it do, through its public entry points.

Three ways in, as programs take them:

* a compiled StableHLO program on device memory (``Client.compile`` at O3, ``Executable.execute_on_device`` on a stream of
  the program's own): inference and training loops that keep their tensors on the GPU;
* the same on host arrays (``Client.buffer`` -> ``Executable.execute`` -> ``Buffer.to_numpy``): a request that arrives from
  and is answered to the host;
* single kernels on CUDA tensors (``metalhlo_b200.cuda``).

``listed()`` names twelve cases, ``draw()`` gives more of the ranges they stand for. One client, one executable per program
text and one stream serve the whole process, as in a serving loop; every state has inputs and outputs of its own.
"""
from __future__ import annotations

import math

import torch

from metalhlo_b200 import capi, cuda, modules
from metalhlo_b200.modules import tt

TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i32": torch.int32}
SIZE = {"f32": 4, "f16": 2, "bf16": 2, "i32": 4}

VOCAB, LAYERS, D_MODEL, HEADS = 50257, 12, 768, 12  # the GPT-2-small architecture of the benchmark

_process = {}


def _client():
    if "client" not in _process:
        _process["client"] = capi.Client()
    return _process["client"]


def _stream():
    if "stream" not in _process:
        _process["stream"] = torch.cuda.Stream()
    return _process["stream"]


# ---- the cases -------------------------------------------------------------------------------------------------------

def listed():
    return [
        # one small request from the host and back: what is left of the latency when there is next to nothing to compute
        dict(name="mlp_host_8x256x256_f32", kind="mlp", host=True, m=8, k=256, n=256, dt="f32"),
        # dense layer + bias + tanh-GELU + softmax in fp32, the configuration the benchmark's baseline names first
        dict(name="mlp_512x1024x1024_f32", kind="mlp", host=False, m=512, k=1024, n=1024, dt="f32"),
        # LayerNorm, RMSNorm and softmax over long rows: the memory-bound side of every transformer
        dict(name="norms_32768x4096_bf16", kind="norms", rows=32768, hidden=4096, dt="bf16"),
        # prefill attention of a large model
        dict(name="attention_8x32x4096x128_bf16", kind="attention", dt="bf16", batch=8, heads=32, seq=4096, head_dim=128, causal=True, program=False),
        # fp32 self-attention as a program of plain operators, the block of the reference's own benchmarks
        dict(name="attention_8x12x512x64_f32", kind="attention", dt="f32", batch=8, heads=12, seq=512, head_dim=64, causal=False, program=True),
        # one large dense product
        dict(name="gemm_8192_bf16", kind="gemm", dt="bf16", batch=1, m=8192, n=8192, k=8192, trans_b=False, bias=False, epilogue="none"),
        # a product whose extents fit no tile and no 16-byte grid, with bias and activation
        dict(name="gemm_1021x3001x1111_f16", kind="gemm", dt="f16", batch=1, m=1021, n=3001, k=1111, trans_b=False, bias=True, epilogue="gelu_tanh"),
        # GPT-2-small forward pass at the benchmark's batch: throughput serving
        dict(name="gpt2_32x1024_f16", kind="gpt2", batch=32, seq=1024, dt="f16"),
        # the same model on one short prompt of odd length: latency serving
        dict(name="gpt2_1x201_f16", kind="gpt2", batch=1, seq=201, dt="f16"),
        # loss and gradients of an embedding + two-layer MLP: the forward and backward half of a training step
        dict(name="train_2048x8192x256_f32", kind="train", tokens=2048, vocab=8192, d=256, hidden=1024, out=128, dt="f32"),
        # residual CNN forward pass on 32 x 32 images
        dict(name="cnn_256x32x64_bf16", kind="cnn", batch=256, size=32, width=64, classes=10, dt="bf16"),
        # argsort of many rows (top-k sampling, ranking): keys in order and their original places
        dict(name="sort_4096x4096_f32", kind="sort", rows=4096, length=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "norms", "attention", "gemm", "gpt2", "train", "cnn", "sort"])
    if kind == "mlp":
        c = dict(kind="mlp", host=rng.random() < 0.5)
        top = 512 if c["host"] else 2048
        c.update(m=_log_int(rng, 1, top), k=_log_int(rng, 64, 2048), n=_log_int(rng, 64, 2048), dt=rng.choice(["f32", "f16"]))
        return c
    if kind == "norms":
        return dict(kind="norms", rows=_log_int(rng, 64, 32768), hidden=_log_int(rng, 64, 4096), dt=rng.choice(["bf16", "f16", "f32"]))
    if kind == "attention":
        dt = rng.choice(["bf16", "f16", "f32"])
        head_dim = rng.choice([64, 128])
        seq = _log_int(rng, 64, 1024 if dt == "f32" else 4096)
        # as much work as the listed cases of the type at most
        most = (8 * 12 * 512 * 512 * 64 if dt == "f32" else 8 * 32 * 4096 * 4096 * 128 // 2) // (seq * seq * head_dim)
        heads = rng.choice([h for h in (1, 2, 4, 8, 12, 16, 32) if h <= max(1, most)])
        batch = _log_int(rng, 1, max(1, min(64, most // heads)))
        return dict(kind="attention", dt=dt, batch=batch, heads=heads, seq=seq, head_dim=head_dim, causal=rng.random() < 0.5, program=rng.random() < 0.5)
    if kind == "gemm":
        dt = rng.choice(["bf16", "f16"])
        if rng.random() < 0.5:  # extents on the 16-byte grid
            m, n, k = (_log_int(rng, 8, 1024) * 8 for _ in range(3))
            batch = 1
        else:
            m, n, k = (_log_int(rng, 33, 3001) for _ in range(3))
            batch = rng.choice([1, 1, 2, 7])
            while batch > 1 and batch * m * n * k > 1021 * 3001 * 1111:
                batch -= 1
            while m * n * k > 2 * 1021 * 3001 * 1111:
                m, n, k = (max(33, v * 3 // 4) for v in (m, n, k))
        bias = batch == 1 and rng.random() < 0.5
        return dict(kind="gemm", dt=dt, batch=batch, m=m, n=n, k=k, trans_b=rng.random() < 0.5, bias=bias,
                    epilogue=rng.choice(["none", "gelu_tanh", "silu", "relu"]) if bias else "none")
    if kind == "gpt2":
        seq = _log_int(rng, 32, 1024)
        return dict(kind="gpt2", batch=_log_int(rng, 1, 32 * 1024 // seq), seq=seq, dt=rng.choice(["f16", "bf16"])) if seq > 256 else \
            dict(kind="gpt2", batch=_log_int(rng, 1, 32), seq=seq, dt=rng.choice(["f16", "bf16"]))
    if kind == "train":
        return dict(kind="train", tokens=_log_int(rng, 128, 2048), vocab=_log_int(rng, 512, 16384), d=_log_int(rng, 32, 512), hidden=_log_int(rng, 64, 1024),
                    out=_log_int(rng, 16, 256), dt="f32")
    if kind == "cnn":
        return dict(kind="cnn", batch=_log_int(rng, 1, 256), size=2 * _log_int(rng, 12, 32), width=8 * _log_int(rng, 2, 16), classes=_log_int(rng, 10, 1000),
                    dt=rng.choice(["bf16", "f16"]))
    length = _log_int(rng, 64, 65536)
    return dict(kind="sort", rows=_log_int(rng, 1, max(1, min(4096, 4096 * 4096 // length))), length=length)


# ---- program texts that the package has no builder for ------------------------------------------------------------------

def _train_text(c):
    """Loss and gradients of mean((tanh(table[ids] . w1 + b1) . w2 + b2 - target)^2) in the forms jax.value_and_grad prints."""
    B, V, D, H, O = c["tokens"], c["vocab"], c["d"], c["hidden"], c["out"]

    def t(*s):
        return tt(s, "f32")

    def dot(out, a, b, ca, cb, ta, tb, to):
        return f"    {out} = stablehlo.dot_general {a}, {b}, contracting_dims = [{ca}] x [{cb}] : ({ta}, {tb}) -> {to}\n"

    body = (
        f"    %zero = stablehlo.constant dense<0.000000e+00> : tensor<f32>\n"
        f"    %one = stablehlo.constant dense<1.000000e+00> : {t(B, H)}\n"
        f"    %idx = stablehlo.reshape %arg0 : (tensor<{B}xi32>) -> tensor<{B}x1xi32>\n"
        f"    %h0 = \"stablehlo.gather\"(%arg1, %idx) <{{dimension_numbers = #stablehlo.gather<offset_dims = [1], collapsed_slice_dims = [0], "
        f"start_index_map = [0], index_vector_dim = 1>, indices_are_sorted = false, slice_sizes = array<i64: 1, {D}>}}> : "
        f"({t(V, D)}, tensor<{B}x1xi32>) -> {t(B, D)}\n"
        + dot("%d1", "%h0", "%arg2", 1, 0, t(B, D), t(D, H), t(B, H)) +
        f"    %b1 = stablehlo.broadcast_in_dim %arg3, dims = [1] : ({t(H)}) -> {t(B, H)}\n"
        f"    %a1 = stablehlo.add %d1, %b1 : {t(B, H)}\n"
        f"    %h1 = stablehlo.tanh %a1 : {t(B, H)}\n"
        + dot("%d2", "%h1", "%arg4", 1, 0, t(B, H), t(H, O), t(B, O)) +
        f"    %b2 = stablehlo.broadcast_in_dim %arg5, dims = [1] : ({t(O)}) -> {t(B, O)}\n"
        f"    %y = stablehlo.add %d2, %b2 : {t(B, O)}\n"
        f"    %diff = stablehlo.subtract %y, %arg6 : {t(B, O)}\n"
        f"    %sq = stablehlo.multiply %diff, %diff : {t(B, O)}\n"
        f"    %sum = stablehlo.reduce(%sq init: %zero) applies stablehlo.add across dimensions = [0, 1] : ({t(B, O)}, tensor<f32>) -> tensor<f32>\n"
        f"    %count = stablehlo.constant dense<{float(B * O):e}> : tensor<f32>\n"
        f"    %loss = stablehlo.divide %sum, %count : tensor<f32>\n"
        f"    %two = stablehlo.constant dense<{2.0 / (B * O):e}> : {t(B, O)}\n"
        f"    %gy = stablehlo.multiply %diff, %two : {t(B, O)}\n"
        + dot("%gw2", "%h1", "%gy", 0, 0, t(B, H), t(B, O), t(H, O)) +
        f"    %gb2 = stablehlo.reduce(%gy init: %zero) applies stablehlo.add across dimensions = [0] : ({t(B, O)}, tensor<f32>) -> {t(O)}\n"
        + dot("%gh1", "%gy", "%arg4", 1, 1, t(B, O), t(H, O), t(B, H)) +
        f"    %hh = stablehlo.multiply %h1, %h1 : {t(B, H)}\n"
        f"    %dh = stablehlo.subtract %one, %hh : {t(B, H)}\n"
        f"    %ga1 = stablehlo.multiply %gh1, %dh : {t(B, H)}\n"
        + dot("%gw1", "%h0", "%ga1", 0, 0, t(B, D), t(B, H), t(D, H)) +
        f"    %gb1 = stablehlo.reduce(%ga1 init: %zero) applies stablehlo.add across dimensions = [0] : ({t(B, H)}, tensor<f32>) -> {t(H)}\n"
        + dot("%gh0", "%ga1", "%arg2", 1, 1, t(B, H), t(D, H), t(B, D)) +
        f"    %zt = stablehlo.constant dense<0.000000e+00> : {t(V, D)}\n"
        f"    %gtable = \"stablehlo.scatter\"(%zt, %idx, %gh0) <{{indices_are_sorted = false, scatter_dimension_numbers = "
        f"#stablehlo.scatter<update_window_dims = [1], inserted_window_dims = [0], scatter_dims_to_operand_dims = [0], index_vector_dim = 1>, "
        f"unique_indices = false}}> ({{\n    ^bb0(%p: tensor<f32>, %q: tensor<f32>):\n      %s = stablehlo.add %p, %q : tensor<f32>\n"
        f"      stablehlo.return %s : tensor<f32>\n    }}) : ({t(V, D)}, tensor<{B}x1xi32>, {t(B, D)}) -> {t(V, D)}")
    return modules.func([f"tensor<{B}xi32>", t(V, D), t(D, H), t(H), t(H, O), t(O), t(B, O)], ["tensor<f32>", t(D, H), t(H), t(H, O), t(O), t(V, D)],
                        body, "%loss, %gw1, %gb1, %gw2, %gb2, %gtable")


def _sort_text(rows, n):
    """Stable ascending sort of every row in the IEEE total order, and the permutation that gives it."""
    t, ti = tt((rows, n), "f32"), tt((rows, n), "i32")
    return (f"func.func @main(%x: {t}) -> ({t}, {ti}) {{\n  %i = stablehlo.iota dim = 1 : {ti}\n"
            f"  %0:2 = \"stablehlo.sort\"(%x, %i) <{{dimension = 1 : i64, is_stable = true}}> ({{\n"
            f"  ^bb0(%a: tensor<f32>, %b: tensor<f32>, %c: tensor<i32>, %d: tensor<i32>):\n"
            f"    %p = stablehlo.compare  LT, %a, %b,  TOTALORDER : (tensor<f32>, tensor<f32>) -> tensor<i1>\n    stablehlo.return %p : tensor<i1>\n"
            f"  }}) : ({t}, {ti}) -> ({t}, {ti})\n  return %0#0, %0#1 : {t}, {ti}\n}}\n")


# ---- inputs ----------------------------------------------------------------------------------------------------------

def _normal(g, shape, dt, scale=1.0, shift=0.0):
    x = torch.randn(shape, device="cuda", dtype=torch.float32, generator=g)
    return x.mul_(scale).add_(shift).to(TORCH[dt])


def _program(text, inputs):
    """State of a compiled program on device memory: its inputs and the outputs it writes."""
    exe = _client().compile(text, opt_level=3)
    codes = {capi.F32: torch.float32, capi.F16: torch.float16, capi.BF16: torch.bfloat16, capi.I32: torch.int32}
    outs = []
    for i in range(exe.output_count):
        shape, code = exe.output_type(i)
        outs.append(torch.empty(shape, dtype=codes[code], device="cuda"))
    _stream().wait_stream(torch.cuda.current_stream())
    return dict(exe=exe, inputs=inputs, outs=outs, in_ptrs=[t.data_ptr() for t in inputs], out_ptrs=[t.data_ptr() for t in outs],
                stream=_stream().cuda_stream)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "mlp":
        m, k, n, dt = case["m"], case["k"], case["n"], case["dt"]
        x, w, b = _normal(g, (m, k), dt), _normal(g, (k, n), dt, 0.02), _normal(g, (n,), dt, 0.02)
        text = modules.mlp_softmax_module(m, k, n, dt)
        if not case["host"]:
            return _program(text, [x, w, b])
        client = _client()
        return dict(exe=client.compile(text, opt_level=3), client=client, x=x.cpu().numpy(), weights=[client.buffer(w), client.buffer(b)])
    if kind == "norms":
        rows, hidden, dt = case["rows"], case["hidden"], case["dt"]
        x = _normal(g, (rows, hidden), dt)
        return _program(modules.norm_sweep_module(rows, hidden, dt), [x, _normal(g, (hidden,), dt, 0.1, 1.0), _normal(g, (hidden,), dt, 0.1)])
    if kind == "attention":
        shape = (case["batch"], case["heads"], case["seq"], case["head_dim"])
        qkv = [_normal(g, shape, case["dt"]) for _ in range(3)]
        if case["program"]:
            return _program(modules.attention_text(*shape, case["dt"], case["causal"])[0], qkv)
        return dict(qkv=qkv, scale=1.0 / math.sqrt(case["head_dim"]), causal=case["causal"])
    if kind == "gemm":
        m, n, k, dt = case["m"], case["n"], case["k"], case["dt"]
        lead = (case["batch"],) if case["batch"] > 1 else ()
        return dict(a=_normal(g, lead + (m, k), dt), b=_normal(g, lead + ((n, k) if case["trans_b"] else (k, n)), dt, 1.0 / math.sqrt(k)),
                    bias=_normal(g, (n,), dt) if case["bias"] else None, epilogue=case["epilogue"], trans_b=case["trans_b"])
    if kind == "gpt2":
        text, params = modules.gpt2_module(batch=case["batch"], seq=case["seq"], layers=LAYERS, d_model=D_MODEL, heads=HEADS, vocab=VOCAB, dt=case["dt"])
        ins = []
        for name, shape, dt in params:
            if dt == "i32":
                ins.append(torch.randint(0, VOCAB, shape, device="cuda", dtype=torch.int32, generator=g))
            elif name.endswith("_g"):
                ins.append(torch.ones(shape, device="cuda"))
            elif name.endswith(("ln1_b", "ln2_b", "lnf_b")):
                ins.append(torch.zeros(shape, device="cuda"))
            else:
                ins.append(_normal(g, shape, "f32", 0.02))
        return _program(text, ins)
    if kind == "train":
        B, V, D, H, O = case["tokens"], case["vocab"], case["d"], case["hidden"], case["out"]
        ins = [torch.randint(0, V, (B,), device="cuda", dtype=torch.int32, generator=g), _normal(g, (V, D), "f32"), _normal(g, (D, H), "f32", 1 / math.sqrt(D)),
               _normal(g, (H,), "f32", 0.1), _normal(g, (H, O), "f32", 1 / math.sqrt(H)), _normal(g, (O,), "f32", 0.1), _normal(g, (B, O), "f32")]
        return _program(_train_text(case), ins)
    if kind == "cnn":
        text, params = modules.cnn_module(batch=case["batch"], size=case["size"], width=case["width"], classes=case["classes"], dt=case["dt"])
        ins = []
        for name, shape, _ in params:
            if name.endswith(("_scale", "_var")):
                ins.append(_normal(g, shape, "f32", 0.1).abs_().add_(0.8))
            elif name == "image":
                ins.append(_normal(g, shape, "f32"))
            else:
                ins.append(_normal(g, shape, "f32", 1.0 / math.sqrt(max(1, math.prod(shape[:-1])))))
        return _program(text, ins)
    return _program(_sort_text(case["rows"], case["length"]), [_normal(g, (case["rows"], case["length"]), "f32")])


# ---- one pass ----------------------------------------------------------------------------------------------------------

def run(state):
    if "weights" in state:
        out, = state["exe"].execute([state["client"].buffer(state["x"])] + state["weights"])
        return out.to_numpy()
    if "qkv" in state:
        return cuda.attention(*state["qkv"], state["scale"], causal=state["causal"])
    if "a" in state:
        return cuda.gemm(state["a"], state["b"], bias=state["bias"], epilogue=state["epilogue"], trans_b=state["trans_b"])
    state["exe"].execute_on_device(state["in_ptrs"], state["out_ptrs"], state["stream"])
    return state["outs"]


# ---- what a pass cannot do without, and how exact it is --------------------------------------------------------------------

def work(case):
    kind, es = case["kind"], SIZE[case.get("dt", "f32")]
    if kind == "mlp":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": es * (m * k + k * n + n + m * n), "flops": 2 * m * k * n}
    if kind == "norms":  # x read once for all three results
        n = case["rows"] * case["hidden"]
        return {"bytes": es * (4 * n + 2 * case["hidden"]), "flops": 16 * n}
    if kind == "attention":
        B, H, S, D = case["batch"], case["heads"], case["seq"], case["head_dim"]
        pairs = S * (S + 1) // 2 if case["causal"] else S * S
        return {"bytes": es * 4 * B * H * S * D, "flops": 4 * B * H * pairs * D}
    if kind == "gemm":
        b, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        return {"bytes": es * (b * (m * k + k * n + m * n) + (n if case["bias"] else 0)), "flops": 2 * b * m * n * k}
    if kind == "gpt2":  # fp32 parameters and ids in, logits out; causal attention at the pairs it needs
        B, S = case["batch"], case["seq"]
        params = VOCAB * D_MODEL + S * D_MODEL + LAYERS * (12 * D_MODEL * D_MODEL + 13 * D_MODEL) + 2 * D_MODEL
        return {"bytes": 4 * params + 4 * B * S + es * B * S * VOCAB,
                "flops": B * S * 2 * (LAYERS * 12 * D_MODEL * D_MODEL + D_MODEL * VOCAB) + LAYERS * B * 4 * (S * (S + 1) // 2) * D_MODEL}
    if kind == "train":
        B, V, D, H, O = case["tokens"], case["vocab"], case["d"], case["hidden"], case["out"]
        weights = D * H + H + H * O + O
        return {"bytes": 4 * (B + min(B, V) * D + V * D + 2 * weights + B * O + 1), "flops": 6 * B * D * H + 6 * B * H * O}
    if kind == "cnn":
        B, S, W, K = case["batch"], case["size"], case["width"], case["classes"]
        h = S // 2
        return {"bytes": 4 * (B * S * S * 3 + 27 * W + 18 * W * W + 8 * W + W * K + K) + es * B * K,
                "flops": 2 * B * (h * h * (27 * W + 18 * W * W) + W * K)}
    n = case["rows"] * case["length"]
    return {"bytes": 12 * n, "flops": 0}


def tolerance(case):
    if case["kind"] == "sort":
        return "exact"
    dt = case["dt"]
    if dt == "f32":
        return {"rel": 1e-5}
    # the result's own rounding is 2^-9 (bf16) or 2^-12 (f16) at worst; programs round their intermediate tensors as well
    return {"rel": 1e-2} if dt == "bf16" or case["kind"] in ("gpt2", "cnn", "attention") else {"rel": 2e-3}
