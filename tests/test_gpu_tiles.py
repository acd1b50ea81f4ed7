"""Edges of the exact small-batch kernel and of the prefill kernel's 384-row tiles, against the oracle."""
import pytest

from tilus_b200 import ops
from tilus_b200.dtypes import weight_dtype

from .test_gpu_parity import _forced

pytestmark = pytest.mark.gpu


# one row past a 256-row tile, the first half's edge (192 rows) and its neighbours, a full tile, one row of the next
@pytest.mark.parametrize("M,N,K,splits", [(257, 272, 1024, 1), (384, 256, 512, 1), (385, 144, 1024, 1),
                                          (576, 128, 512, 1), (577, 400, 1152, 1), (784, 256, 512, 1),
                                          (768, 256, 2048, 4)])
@pytest.mark.parametrize("w,zp,group", [("uint4b", 8, 128), ("float6_e3m2", 0, 64), ("int8", 0, 32)])
def test_prefill_384_row_tiles(M, N, K, splits, w, zp, group):
    m_tiles, n_tiles = (M + 383) // 384, (N + 127) // 128
    _forced(M, N, K, weight_dtype(w), zp, dict(kernel=1, splits=splits, tile_m=384, m_tiles=m_tiles,
                                               ctas_per_split=m_tiles * n_tiles), seed=M, group=group)


def test_prefill_384_row_tiles_are_planned_and_walked():
    """More tiles than SMs: accumulators and both rings carry over tile boundaries."""
    M, N, K = 1000, 12304, 256
    dt = weight_dtype("uint4b")
    assert ops.plan(M, N, K, dt, 8, 128)["tile_m"] == 384
    _forced(M, N, K, dt, 8, dict(), seed=3)


# 5 .. 16 rows; one column tile and ragged ones; one 128-row group, and more groups than a CTA's run; one scale per
# group, per several groups and per column
@pytest.mark.parametrize("M", [5, 8, 9, 16])
@pytest.mark.parametrize("N,K,group", [(16, 128, 128), (272, 1024, 512), (144, 8192, 8192), (4112, 2048, 128)])
@pytest.mark.parametrize("w,zp", [("uint4b", 8), ("int8", 0), ("float6_e3m2", 0), ("uint1b", 0)])
def test_exact_small_batch_kernel(M, N, K, group, w, zp):
    """By the plan of 16 rows, which is always the exact kernel's (some batches of 5..8 rows go to the stream kernel)."""
    pl = ops.plan(16, N, K, weight_dtype(w), zp, group)
    assert pl["tile_m"] == 16
    plan = {f: pl[f] for f in ("kernel", "splits", "cluster", "ctas_per_split", "tile_m", "stages")}
    plan["resident"] = 0  # (nor to the one that keeps the activations in registers)
    _forced(M, N, K, weight_dtype(w), zp, plan, seed=M + N, group=group)


@pytest.mark.parametrize("M", [2, 4])
def test_few_rows_whose_stream_plan_cuts_k(M):
    """448 column tiles have no divisor near two CTAs per SM: the exact kernel takes them from two rows on."""
    dt = weight_dtype("uint4b")
    assert ops.plan(1, 7168, 2048, dt, 8, 128)["tile_m"] == 0 and ops.plan(M, 7168, 2048, dt, 8, 128)["tile_m"] == 16
    for plan in (dict(), dict(resident=0)):  # the kernel that keeps the activations in registers takes fp16 there
        _forced(M, 7168, 2048, dt, 8, plan, seed=M)


@pytest.mark.parametrize("w,zp", [("uint8", 128), ("int8", 0), ("int6b", 0), ("uint4b", 8), ("uint1b", 1)])
def test_exact_small_batch_kernel_keeps_the_bits_of_its_sums(w, zp):
    """Activations away from zero: the zero point is subtracted while the products are summed, so the fp32 sums
    stay near their results.  An MMA loses at most 2^-23 of the running sum; 512 of them (16 per 128 rows, 32 groups), as
    a random walk, 22.6 * 2^-23 of it.  With the running sum no larger than the result, a result within
    that distance of the middle between two fp16 values (2^-11 apart) may go to the other one: 2 * 22.6 * 2^-23 / 2^-11 =
    1.1 % of the outputs.  (Zero points subtracted at the end of a group: 6.3 % for 8 bits.)"""
    import torch
    from oracle import quant_oracle as qo
    from tilus_b200 import packing

    m, n, k, group, dt = 8, 1024, 4096, 128, weight_dtype(w)
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(1)
    codes = torch.randint(0, 1 << dt.nbits, (k, n), device=dev, generator=gen, dtype=torch.int32).to(torch.uint8)
    a = (torch.randn(m, k, device=dev, generator=gen) + 3.0).half()
    sc = (torch.rand(k // group, n, device=dev, generator=gen) * 0.01 + 0.002).half()
    plan = dict(kernel=2, tile_m=16, splits=1, cluster=1, ctas_per_split=128, resident=0)
    got = ops.quantized_matmul(a, packing.interleave(codes, dt).to(dev), sc, dt, group, zp, plan_override=plan)
    value = torch.from_numpy(qo.decode_table(dt)).to(dev)[codes.long()] - zp
    ref = a.double() @ (value * sc.double().repeat_interleave(group, 0))
    assert float((got != ref.half()).float().mean()) <= 0.011
