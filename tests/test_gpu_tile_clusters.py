"""The small-batch kernel with a cluster of CTAs per column tile: what the CTAs send each other, and rings that make room for it."""
import pytest
import torch

from tilus_b200 import dtypes as D
from tilus_b200 import ops

pytestmark = pytest.mark.gpu


def _check(M, N, K, dt, zp, group, cluster, act=torch.float16):
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(M * 7 + cluster)
    bq = torch.randint(0, 256, (N * K * dt.nbits // 8,), dtype=torch.uint8, device=dev, generator=gen)
    sc = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).to(act)
    a = torch.randn(M, K, device=dev, generator=gen).to(act)
    ref = a.double() @ ops.dequantize(bq, sc, dt, group, zp).double()  # the weights that the kernel multiplies by
    tiles = (N + 127) // 128
    ws = torch.zeros(ops.workspace_bytes(M, N, K, dt, zp, group), dtype=torch.uint8, device=dev)
    plan = dict(kernel=3, tile_m=(M + 15) // 16 * 16, splits=1, cluster=cluster, ctas_per_split=tiles * cluster, resident=0)
    outs = [ops.quantized_matmul(a, bq, sc, dt, group, zp, workspace=ws, plan_override=plan) for _ in range(20)]
    # one rounding of the output (2^-11, bfloat16 2^-8) and the fp32 sums
    eps = 2.0 ** -11 if act == torch.float16 else 2.0 ** -8
    assert bool(((outs[0].double() - ref).abs() <= eps * ref.abs() + 2e-5 * ref.abs().max()).all())
    for c in outs[1:]:  # calls that overlap on the GPU; the CTAs' sums are added in order
        assert torch.equal(c, outs[0])
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("cluster", [2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("M", [33, 36, 49, 64, 65, 100, 128])
def test_rows_over_clusters(M, cluster):
    """Quads of rows that do not divide among the CTAs, owners without rows, the last one with fewer."""
    _check(M, 400, 2176, D.uint4b, 8, 128, cluster)


@pytest.mark.parametrize("dt,zp,group", [(D.uint8, 128, 32), (D.int6b, 0, 64), (D.uint2b, 2, 128), (D.float6_e3m2, 0, 1024)], ids=str)
@pytest.mark.parametrize("M,act", [(128, torch.float16), (112, torch.bfloat16), (40, torch.bfloat16)], ids=str)
def test_rings_beside_the_sums(M, dt, zp, group, act):
    """8-bit weights with scales per 32 rows next to 128 rows of activations: the shallowest rings."""
    _check(M, 272, 2048, dt, zp, group, 4, act)


@pytest.mark.parametrize("M", [9, 17, 32])
def test_clusters_of_few_rows_by_an_edited_plan(M):
    """Up to 16 rows the exact kernel's clusters, up to 32 a form that no plan has."""
    _check(M, 1040, 2048, D.int4b, 0, 64, 4)


@pytest.mark.parametrize("M,N,K,dt,group,act", [
    (40, 36864, 512, D.uint4b, 128, torch.float16),   # 288 column tiles, two for each of 144 CTAs
    (17, 20000, 512, D.uint4b, 128, torch.float16),   # 157 tiles, whole ones, 79 CTAs of which one has a single tile
    (32, 16384, 1024, D.uint2b, 128, torch.float16),  # 128 whole tiles, two CTAs to an SM
    (65, 2064, 1024, D.int6b, 64, torch.bfloat16),    # one tile per CTA beyond 64 rows: three sets, one accumulator
    (128, 1168, 2048, D.uint8, 64, torch.float16),    # the same with a ring too short for three sets
    (24, 4112, 2048, D.int8, 128, torch.float16),     # few rows of a wide type: three sets, the SM to itself
    (32, 2064, 8192, D.float6_e3m2, 8192, torch.bfloat16),
    (9, 1040, 1152, D.int3b, 32, torch.float16)], ids=str)
def test_whole_tiles_and_sets(M, N, K, dt, group, act):
    """Splits of the planned launches where CTAs have whole column tiles, and the number of dequantizing sets."""
    dev = torch.device("cuda:0")
    zp = 1 << (dt.nbits - 1) if dt.kind == D.KIND_UINT else 0
    gen = torch.Generator(device=dev).manual_seed(M)
    bq = torch.randint(0, 256, (N * K * dt.nbits // 8,), dtype=torch.uint8, device=dev, generator=gen)
    sc = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).to(act)
    a = torch.randn(M, K, device=dev, generator=gen).to(act)
    ref = a.double() @ ops.dequantize(bq, sc, dt, group, zp).double()
    ws = torch.zeros(ops.workspace_bytes(M, N, K, dt, zp, group), dtype=torch.uint8, device=dev)
    outs = [ops.quantized_matmul(a, bq, sc, dt, group, zp, workspace=ws) for _ in range(10)]
    eps = 2.0 ** -11 if act == torch.float16 else 2.0 ** -8  # as above
    assert bool(((outs[0].double() - ref).abs() <= eps * ref.abs() + 2e-5 * ref.abs().max()).all())
    for c in outs[1:]:
        assert torch.equal(c, outs[0])
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("M,N,K,dt,group,act,ctas,cluster", [
    (12, 6144, 4096, D.float8_e5m2, 64, torch.bfloat16, 96, 2), (32, 6144, 4096, D.int8, 128, torch.float16, 96, 2),
    (24, 8192, 4096, D.float6_e3m2, 128, torch.float16, 128, 2), (32, 20480, 512, D.int8, 128, torch.float16, 80, 1),
    (24, 11008, 4096, D.int8, 128, torch.float16, 148, 1), (24, 14336, 8192, D.int3b, 128, torch.float16, 148, 1)], ids=str)
def test_splits_of_types_with_an_sm_to_themselves(M, N, K, dt, group, act, ctas, cluster):
    """Up to 32 rows: the form that was the fastest of those forced at these shapes."""
    pl = ops.plan(M, N, K, dt, 0, group, act_dtype=act)
    assert (pl["ctas_per_split"], pl["cluster"]) == (ctas, cluster)
