"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one pass through the public entry points: single linears from the smallest decode call to
prefill, the linears of a decode step of a whole model (called one by one, or replayed from a CUDA
graph as a serving program does), calls on host buffers, a gate_up projection with the SwiGLU and
the FP8 cast behind it, and loading a layer from dense weights.
"""
from __future__ import annotations

import math

import torch

from tilus_b200 import QuantizedLinear
from tilus_b200.dtypes import KIND_UINT, weight_dtype

DEVICE = "cuda"
TORCH_ACT = {"float16": torch.float16, "bfloat16": torch.bfloat16}


def listed():
    return [
        # The smallest call: one decode token through one 4096 x 4096 layer with 3-bit weights and one
        # scale per channel.  Nearly all of it is call and launch latency.
        _linear("decode_m1_i3_4096", 1, 4096, 4096, "int3b", 4096),
        # The benchmark's headline decode shape, a few layers in a row (their weights exceed L2).
        _linear("decode_m1_u4_8192", 1, 8192, 8192, "uint4b", 128, layers=6),
        # A decode step of a Llama-3-8B-shaped model, one sequence, captured once and replayed.
        _stack("step_m1_graph", 1, layers=32, graph=True),
        # The same step for eight sequences in a program that calls the layers one by one.
        _stack("step_m8_calls", 8, layers=32, graph=False),
        # A decode batch of 16 with 6-bit float weights, per-channel scales.
        _linear("decode_m16_f6_4096", 16, 4096, 4096, "float6_e3m2", 4096, layers=8),
        # A decode step for 64 sequences, replayed.
        _stack("step_m64_graph", 64, layers=32, graph=True),
        # A ragged batch in bfloat16: 6-bit weights, scales per 64 rows, sizes that fill no tile evenly.
        _linear("batch_m100_i6_bf16", 100, 11008, 4224, "int6b", 64, act="bfloat16", layers=3),
        # Prompt processing with one row more than whole tiles (the reference example times 4096 and 4097).
        _linear("prefill_m4097_f4_bf16", 4097, 12288, 4096, "float4_e2m1", 128, act="bfloat16"),
        # The largest: prefill of a 70B-class MLP-up projection.
        _linear("prefill_m4096_i4_28672", 4096, 28672, 8192, "int4b", 128),
        # Decode called by a program that keeps activations and results in pinned host memory.
        _linear("host_m1_u4_8192", 1, 8192, 8192, "uint4b", 128, layers=6, op="host"),
        # gate_up projection with SwiGLU and the per-token FP8 cast behind it, a decode batch.
        dict(name="gate_up_cast_m8_u4", op="gate_up_cast", m=8, n=28672, k=4096, w="uint4b", group=128, act="float16",
             clamp=False, layers=2),
        # Loading: a dense gate_up weight is quantized and packed.
        dict(name="quantize_i4_28672x4096", op="quantize", n=28672, k=4096, w="int4b", group=128, act="float16"),
    ]


def _linear(name, m, n, k, w, group, act="float16", layers=1, op="linear"):
    return dict(name=name, op=op, m=m, n=n, k=k, w=w, group=group, act=act, layers=layers)


def _stack(name, m, layers, graph, hidden=4096, qkv=6144, ffn=14336):
    return dict(name=name, op="stack", m=m, hidden=hidden, qkv=qkv, ffn=ffn, layers=layers, graph=graph, w="uint4b",
                group=128, act="float16")


WEIGHTS = ["uint4b", "uint4b", "int4b", "int4b", "int8", "uint8", "int6b", "uint6b", "int3b", "uint3b", "uint2b", "uint1b",
           "float8_e5m2", "float6_e3m2", "float4_e2m1", "float3_e1m1"]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["linear", "stack", "host", "gate_up_cast", "quantize"], [11, 3, 2, 2, 2])[0]
    act = rng.choice(["float16", "float16", "bfloat16"])
    w = rng.choice(WEIGHTS)
    if op == "stack":
        hidden = 512 * rng.randint(2, 10)
        case = _stack("", _log_int(rng, 1, 96), rng.randint(4, 32), rng.random() < 0.5, hidden,
                      hidden + 128 * rng.randint(2, 16), 256 * rng.randint(hidden // 128, hidden // 64))
        case.pop("name")
        return case
    # every other K is a multiple of 512, the others of 128 only; N of 256 or of 16 only
    k = max(1024, 512 * round(_log_int(rng, 1024, 14336) / 512)) if rng.random() < 0.5 else 128 * (_log_int(rng, 1024, 14336) // 128)
    n = 256 * max(4, _log_int(rng, 1024, 28672) // 256) if rng.random() < 0.5 else 16 * (_log_int(rng, 1024, 28672) // 16)
    group = rng.choice([128, 128, 128, 128, 32, 64, 256, k])
    if k % group:
        group = 128
    if op == "quantize":
        w = rng.choice(["int4b", "int8", "int6b", "int3b", "float6_e3m2", "float4_e2m1"])
        return dict(op=op, n=n, k=k, w=w, group=group, act=act)
    if op == "host":
        m = _log_int(rng, 1, 64)
    elif op == "gate_up_cast":
        m, n = _log_int(rng, 1, 512), 256 * max(4, n // 256)
    else:
        m = _log_int(rng, 1, 4608)
        m = max(1, min(m, int(1.5e12 / (2.0 * n * k))))
    if group < 128 and weight_dtype(w).nbits == 8:
        group = 128  # 8-bit weights are used with scales per 128 rows or more
    layers = 1 if m > 128 else rng.randint(1, 4)
    case = dict(op=op, m=m, n=n, k=k, w=w, group=group, act=act, layers=layers)
    if op == "gate_up_cast":
        case["clamp"] = rng.random() < 0.5
    return case


# ---- inputs ---------------------------------------------------------------------------------------------
def _code_rms(dt):
    """Root mean square of the values of uniformly drawn codes."""
    if not dt.is_float():
        return math.sqrt(((1 << dt.nbits) ** 2 - 1) / 12.0 + 0.25)
    if dt.exponent_nbits == 5:
        return 0.4  # exponents 0..15 only, see _packed
    e, m, bias = dt.exponent_nbits, dt.mantissa_nbits, dt.exponent_bias
    values = []
    for code in range(1 << (e + m)):
        ex, ma = code >> m, (code & ((1 << m) - 1)) / (1 << m)
        values.append(ma * 2.0 ** (1 - bias) if ex == 0 else (1 + ma) * 2.0 ** (ex - bias))
    return math.sqrt(sum(v * v for v in values) / len(values))


def _packed(dt, n, k, gen, zero_mean=False):
    """Packed weights with uniformly drawn codes: every bit pattern of the packed bytes is one."""
    size = n * k * dt.nbits // 8
    if zero_mean:  # 4-bit codes 1..15, zero mean around the zero point 8: keeps a long chain of layers in range
        lo = torch.randint(1, 16, (size,), dtype=torch.uint8, device=DEVICE, generator=gen)
        return lo + 16 * torch.randint(1, 16, (size,), dtype=torch.uint8, device=DEVICE, generator=gen)
    data = torch.randint(0, 256, (size,), dtype=torch.uint8, device=DEVICE, generator=gen)
    if dt.is_float() and dt.exponent_nbits == 5:
        data &= 0xBF  # magnitudes below 2: no Inf / NaN patterns, and products that stay inside fp16
    return data


def _layer(dt, n, k, group, act, gen, zero_mean=False):
    zero_point = 1 << (dt.nbits - 1) if dt.kind == KIND_UINT else 0
    with torch.device(DEVICE):
        layer = QuantizedLinear(act, dt, group, k, n, zero_point=zero_point)
    # scales that keep the outputs about as large as the inputs
    mean = 1.0 / (math.sqrt(k) * _code_rms(dt))
    scales = (torch.rand(k // group, n, device=DEVICE, generator=gen) * 0.5 + 0.75) * mean
    layer.load_packed(_packed(dt, n, k, gen, zero_mean), scales.to(TORCH_ACT[act]), layout="b200")
    return layer


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    op, act = case["op"], case["act"]
    dt, group = weight_dtype(case["w"]), case["group"]

    def rows(m, k):
        return torch.randn(m, k, device=DEVICE, generator=gen).to(TORCH_ACT[act])

    state = dict(op=op)
    if op == "quantize":
        state["weight"] = (torch.randn(case["n"], case["k"], device=DEVICE, generator=gen) * 0.02).to(TORCH_ACT[act])
        with torch.device(DEVICE):
            state["layer"] = QuantizedLinear(act, dt, group, case["k"], case["n"])
        return state
    if op == "stack":
        h, q, f = case["hidden"], case["qkv"], case["ffn"]
        state["blocks"] = [[_layer(dt, n, k, group, act, gen, zero_mean=True)
                            for n, k in ((q, h), (h, h), (2 * f, h), (h, f))] for _ in range(case["layers"])]
        state["x"] = rows(case["m"], h)
        state["sizes"] = (h, f)
        state["graph"] = None
        if case["graph"]:
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                _step(state)  # one plain call before the capture
            torch.cuda.current_stream().wait_stream(stream)
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"], stream=stream):
                state["out"] = _step(state)
        return state
    state["layers"] = [_layer(dt, case["n"], case["k"], group, act, gen) for _ in range(case["layers"])]
    state["x"] = [rows(case["m"], case["k"]) for _ in range(case["layers"])]
    if op == "host":
        state["x"] = [x.cpu().pin_memory() for x in state["x"]]
        state["out"] = [torch.zeros(case["m"], case["n"], dtype=TORCH_ACT[act]).pin_memory() for _ in state["x"]]
    if op == "gate_up_cast":
        state["clamp"] = 1.0 if case["clamp"] else None
    return state


def _step(state):
    """The linears of one decode step, each on the output of the one before it; every block's output."""
    h, f = state["sizes"]
    x, out = state["x"], []
    for qkv, o, gate_up, down in state["blocks"]:
        y = qkv(x)
        y = o(y[:, :h])
        y = gate_up(y)
        x = down(y[:, :f])
        out.append(x)
    return out


def run(state):
    op = state["op"]
    if op == "linear":
        return [layer(x) for layer, x in zip(state["layers"], state["x"])]
    if op == "stack":
        if state["graph"] is None:
            return _step(state)
        state["graph"].replay()
        return state["out"]
    if op == "host":
        return [layer.forward_host(x, y) for layer, x, y in zip(state["layers"], state["x"], state["out"])]
    if op == "gate_up_cast":
        return [layer.forward_swiglu_cast(x, 128, state["clamp"]) for layer, x in zip(state["layers"], state["x"])]
    state["layer"].load_and_quantize(state["weight"])
    return [state["layer"].quantized_weight.data, state["layer"].scales.data]


# ---- what a pass cannot do without, and how far two correct results may be apart --------------------------
def _gemm_work(m, n, k, nbits, group):
    return k * n * nbits / 8 + (k // group) * n * 2 + m * k * 2 + m * n * 2, 2.0 * m * n * k


def work(case):
    b, g = weight_dtype(case["w"]).nbits, case["group"]
    if case["op"] == "quantize":
        n, k = case["n"], case["k"]
        return {"bytes": n * k * 2 + n * k * b / 8 + (k // g) * n * 2, "flops": 2.0 * n * k}
    if case["op"] == "stack":
        h, q, f = case["hidden"], case["qkv"], case["ffn"]
        parts = [_gemm_work(case["m"], n, k, b, g) for n, k in ((q, h), (h, h), (2 * f, h), (h, f))]
    else:
        parts = [_gemm_work(case["m"], case["n"], case["k"], b, g)]
    if case["op"] == "gate_up_cast":
        m, hid = case["m"], case["n"] // 2
        parts.append((m * hid + m * (hid // 128) * 4, 8.0 * m * hid))
    return {"bytes": case["layers"] * sum(p[0] for p in parts), "flops": case["layers"] * sum(p[1] for p in parts)}


def tolerance(case):
    if case["op"] == "quantize":
        return "exact"  # codes and scales are defined bit for bit
    if case["op"] == "gate_up_cast":
        # e4m3 steps are 1/8 of a binade: a last-bit difference of the projection moves about one value in
        # a hundred (fp16; ten in bf16) to the neighbouring code
        return {"rel": 1e-2 if case["act"] == "float16" else 2.5e-2, "max": 0.5}
    if case["op"] == "stack":
        return {"rel": 1e-2}  # up to 128 linears in sequence, each rounding weights and outputs to fp16
    # one rounding of each weight and one of each output to the activation dtype
    return {"rel": 2e-3} if case["act"] == "float16" else {"rel": 1e-2}
