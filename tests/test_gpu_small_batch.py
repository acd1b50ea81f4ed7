"""The small-batch kernel where a CTA's run covers several short column tiles, in launches queued back to back."""
import pytest
import torch

from tilus_b200 import dtypes as D
from tilus_b200 import ops

from .launches import kernels
from .test_gpu_parity import _forced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [20, 64, 100, 128])
@pytest.mark.parametrize("N,K", [(28672, 512), (32000, 256), (128256, 256), (18944, 768), (20480, 128)])
def test_runs_of_many_short_tiles_without_synchronisation(M, N, K):
    """Few 128-row groups per column tile: the warps that decode weights reach the end of their CTA's run while
    the MMAs of its first tiles still wait for the launch before.  Twelve launches in a row without a
    synchronisation, four weights, every output compared in full with an fp32 product of the dequantized weights
    (bit-exact with the oracle, test_gpu_parity.py).  One rounding of the output is 2^-11 of its size, sums
    of up to 768 fp32 products stay far below it: 2e-3 of the largest output."""
    dev = torch.device("cuda:0")
    dt, group = D.int4b, 128
    gen = torch.Generator(device=dev).manual_seed(N + K + M)
    layers = []
    for _ in range(4):
        bq = torch.randint(0, 256, (N * K // 2,), dtype=torch.uint8, device=dev, generator=gen)
        scales = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).half()
        layers.append((bq, scales))
    xs = [torch.randn(M, K, device=dev, generator=gen).half() for _ in range(3)]
    pl = ops.plan(M, N, K, dt, 0, group)
    assert pl["kernel"] == 3
    torch.cuda.synchronize()
    outs = [ops.quantized_matmul(xs[i % 3], *layers[i % 4], dt, group) for i in range(12)]
    torch.cuda.synchronize()
    for i, got in enumerate(outs):
        w = ops.dequantize(*layers[i % 4], dt, group).float()
        ref = xs[i % 3].float() @ w
        assert float((got.float() - ref).abs().max()) <= 2e-3 * float(ref.abs().max()), i
    assert ops.device_status(ops.get_workspace(dev, 1 << 20)) == [0, 0, 0, 0]


@pytest.mark.parametrize("M,group", [(5, 128), (16, 512), (24, 128), (64, 32), (128, 128)])
@pytest.mark.parametrize("tiles,ctas", [(7, 3), (9, 9), (10, 9), (23, 4), (8, 4), (41, 40)])
@pytest.mark.parametrize("K", [2048, 2176])
def test_runs_of_one_to_six_column_tiles(M, group, tiles, ctas, K):
    """At least as many column tiles as CTAs: runs that are whole tiles, runs that begin and end inside one, runs one group
    longer than a tile, and a last column tile of 16 columns."""
    if K % group:
        pytest.skip("group does not divide K")
    N, dt = tiles * 128 - 112, D.int4b
    exact = M <= 16 and group % 128 == 0
    plan = dict(kernel=2 if exact else 3, tile_m=16 if exact else 128, splits=1, cluster=1, ctas_per_split=ctas, resident=0)
    _forced(M, N, K, dt, 0, plan, seed=M + tiles, group=group)


@pytest.mark.parametrize("M,dt,group", [(8, D.uint4b, 128), (16, D.int3b, 128), (24, D.uint4b, 128), (64, D.uint4b, 128),
                                        (128, D.int4b, 64)], ids=str)
@pytest.mark.parametrize("N,K", [(28672, 4096), (19072, 4096)])
def test_wide_layers_repeat_their_results_bit_for_bit(M, dt, group, N, K):
    """With at least as many column tiles as CTAs no run is shorter than a tile, so that two CTAs at most add to a tile: whichever
    comes first, the sum of two numbers is the same."""
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(M)
    bq = torch.randint(0, 256, (N * K * dt.nbits // 8,), dtype=torch.uint8, device=dev, generator=gen)
    scales = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).half()
    x = torch.randn(M, K, device=dev, generator=gen).half()
    zp = 8 if dt.kind == D.KIND_UINT else 0
    assert ops.plan(M, N, K, dt, zp, group)["tile_m"] == (M + 15) // 16 * 16
    for plan in (None, dict(resident=0)):
        outs = [ops.quantized_matmul(x, bq, scales, dt, group, zp, plan_override=plan) for _ in range(12)]
        for c in outs[1:]:
            assert torch.equal(c, outs[0])
    call = lambda: ops.quantized_matmul(x, bq, scales, dt, group, zp, plan_override=plan)  # noqa: E731
    assert kernels(call) == ["exact_kernel"] if M <= 16 else kernels(call)[0] in ("batch_kernel", "tile_run_kernel")
