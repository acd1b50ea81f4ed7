"""Calls whose route the plan decides, against the oracle's arithmetic."""
import pytest
import torch

from tilus_b200 import _lib, packing, synth
from tilus_b200 import dtypes as D
from tilus_b200 import ops

from .launches import kernels

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
    force = lambda pl, res=0: ops.quantized_matmul(a, bq, sc, dt, group, plan_override={**{f: pl[f] for f in fields}, "resident": res})  # noqa: E731
    assert close(force(exact_plan), exact) and close(force(exact_plan, 1), exact)
    assert close(force(stream_plan), saturated) and close(force(stream_plan, 1), saturated)
    assert close(ops.quantized_matmul(a, bq, sc, dt, group), saturated)
    assert kernels(lambda: force(exact_plan), lambda: force(exact_plan, 1), lambda: force(stream_plan), lambda: force(stream_plan, 1)) == [
        "exact_kernel", "exact_kernel", "stream_kernel", "resident_kernel"]


@pytest.mark.parametrize("M,N,K", [(8, 129280, 512), (16, 129280, 512), (300, 9472, 1024), (326, 6000, 2048)])
def test_static_workspace_where_the_plan_asks_for_more(M, N, K):
    """Problems whose plan wants more than the built-in scratch and that run without it: whole column tiles in the
    exact kernel, tiles of 256 rows instead of 384 in the prefill kernel.  Twice, on the scratch the first one left."""
    dev = torch.device("cuda:0")
    lib, dt, group = _lib.load(), D.int4b, 128
    gen = torch.Generator(device=dev).manual_seed(M)
    bq = torch.randint(0, 256, (N * K // 2,), dtype=torch.uint8, device=dev, generator=gen)
    sc = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).half()
    a = torch.randn(M, K, device=dev, generator=gen).half()
    assert lib.b200q_workspace_bytes(M, N, K, dt.code, 0, group) > lib.b200q_static_workspace_limit()
    outs = [torch.full((M, N), float("nan"), dtype=torch.float16, device=dev) for _ in range(2)]
    for c in outs:
        _lib.check(lib.b200q_gemm_static_ws(a.data_ptr(), K, bq.data_ptr(), sc.data_ptr(), c.data_ptr(), N, M, N, K,
                                            dt.code, 0, group, _lib.ACT_F16, torch.cuda.current_stream().cuda_stream))
    ref = a.float() @ ops.dequantize(bq, sc, dt, group).float()
    for c in outs:  # one rounding of the output (2^-11) and of each weight (2^-11, exact kernel: none), see also test_gpu_small_batch.py
        assert float((c.float() - ref).abs().max()) <= 2e-3 * float(ref.abs().max())
    assert ops.device_status(None, dev) == [0, 0, 0, 0]


@pytest.mark.parametrize("M", [1, 3, 5, 9, 16])
@pytest.mark.parametrize("N,K", [(272, 1024), (4112, 2048)])
@pytest.mark.parametrize("gap", [1, 4, 6])
def test_decode_batches_write_rows_at_any_distance(M, N, K, gap):
    """Outputs that are columns of a wider tensor whose rows are not a multiple of 16 bytes apart; the columns
    beside them stay untouched."""
    dev = torch.device("cuda:0")
    dt, group = D.uint4b, 128
    prob = synth.make_problem(M, N, K, dt, group, seed=M)
    wide = torch.full((M, N + gap), 7.0, dtype=torch.float16, device=dev)
    bq = packing.interleave(prob["codes"], dt).to(dev)
    a, sc = prob["a"].to(dev), prob["scales"].to(dev)
    ops.quantized_matmul(a, bq, sc, dt, group, 8, out=wide[:, :N])
    ref = a.float() @ ops.dequantize(bq, sc, dt, group, 8).float()
    assert float((wide[:, :N].float() - ref).abs().max()) <= 2e-3 * float(ref.abs().max())
    assert bool((wide[:, N:] == 7.0).all())


@pytest.mark.parametrize("M", [129, 200, 385])
def test_small_batch_kernel_forced_beyond_its_rows(M):
    """A plan edited to kernel 3 for more rows than one launch takes runs in pieces."""
    from .test_gpu_parity import _forced

    _forced(M, 272, 1024, D.int4b, 0, dict(kernel=3, splits=2, ctas_per_split=2), seed=M)


@pytest.mark.parametrize("M", [7, 9, 16])
@pytest.mark.parametrize("N,K,splits", [(272, 1024, 2), (6144, 2048, 4), (6144, 4096, 2)])
@pytest.mark.parametrize("dt", [D.int4b, D.int8, D.float6_e3m2], ids=lambda d: d.name)
def test_k_chunks_put_into_a_decode_plan(M, N, K, splits, dt):
    """The number of k chunks is the one field that an edited decode plan of 5..16 rows needs."""
    from .test_gpu_parity import _forced

    assert ops.plan(M, N, K, dt, 0, 128)["tile_m"] == 16
    _forced(M, N, K, dt, 0, dict(splits=splits), seed=M)


@pytest.mark.parametrize("M,N,K", [(300, 6000, 1024), (329, 9280, 1024)])
def test_prefill_with_less_scratch_than_its_plan_asks_for(M, N, K):
    """A fixed workspace that holds what tiles of 256 rows need, where the plan's tiles of 384 rows would cut K."""
    dev = torch.device("cuda:0")
    dt, group = D.int4b, 128
    gen = torch.Generator(device=dev).manual_seed(M)
    bq = torch.randint(0, 256, (N * K // 2,), dtype=torch.uint8, device=dev, generator=gen)
    sc = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).half()
    a = torch.randn(M, K, device=dev, generator=gen).half()
    pl = ops.plan(M, N, K, dt, 0, group)
    assert pl["tile_m"] == 384 and pl["workspace_bytes"] > (1 << 16)
    ws = torch.zeros(1 << 16, dtype=torch.uint8, device=dev)
    ref = a.float() @ ops.dequantize(bq, sc, dt, group).float()
    c = ops.quantized_matmul(a, bq, sc, dt, group, workspace=ws)
    assert float((c.float() - ref).abs().max()) <= 2e-3 * float(ref.abs().max())
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("M", [20, 37, 80, 100])
@pytest.mark.parametrize("K", [2048, 5120])  # 5120 columns of the activations do not fit the stream kernel in one chunk
def test_small_batch_plans_put_on_another_kernel(M, K, kernel):
    """The kernel is the one field that needs to change: the prefill kernel takes the tile that holds the plan's rows, the
    stream kernel rings, chunks and CTAs that fit it."""
    from .test_gpu_parity import _forced

    assert ops.plan(M, 1920, K, D.int8, 0, 128)["kernel"] == 3
    _forced(M, 1920, K, D.int8, 0, dict(kernel=kernel), seed=M)
