"""Calls whose route the plan decides, against the oracle's arithmetic."""
import pytest
import torch

from tilus_b200 import _lib, packing, synth
from tilus_b200 import dtypes as D
from tilus_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [5, 8])
def test_bf16_runs_the_form_its_plan_names(M):
    """The exact kernel multiplies bfloat16 activations as they are, the stream kernel in fp16 (magnitudes beyond
    65504 saturate): a forced plan is obeyed for bfloat16 too, and the unplanned call runs the reported one."""
    dev = torch.device("cuda:0")
    dt, group, N, K = D.int4b, 128, 512, 1024
    prob = synth.make_problem(M, N, K, dt, group, seed=M)
    a = (prob["a"].float() * 1e5).to(torch.bfloat16).to(dev)
    sc = prob["scales"].to(torch.bfloat16).to(dev)
    bq = packing.interleave(prob["codes"], dt).to(dev)
    w = ops.dequantize(bq, sc, dt, group).double()
    exact, saturated = a.double() @ w, a.double().clamp(-65504, 65504) @ w

    def close(c, ref):
        return float((c.double() - ref).abs().max() / ref.abs().max()) <= 1e-2

    stream_plan = ops.plan(M, N, K, dt, 0, group, act_dtype=torch.bfloat16)
    exact_plan = ops.plan(16, N, K, dt, 0, group)
    assert stream_plan["tile_m"] == 0 and exact_plan["tile_m"] == 16
    fields = ("kernel", "splits", "cluster", "ctas_per_split", "tile_m", "stages")
    force = lambda pl: ops.quantized_matmul(a, bq, sc, dt, group, plan_override={f: pl[f] for f in fields})  # noqa: E731
    assert close(force(exact_plan), exact)
    assert close(force(stream_plan), saturated)
    assert close(ops.quantized_matmul(a, bq, sc, dt, group), saturated)
