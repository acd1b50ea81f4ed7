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
    _forced(M, N, K, weight_dtype(w), zp, dict(), seed=M + N, group=group)


@pytest.mark.parametrize("M", [2, 4])
def test_few_rows_whose_stream_plan_cuts_k(M):
    """448 column tiles have no divisor near two CTAs per SM: the exact kernel takes them from two rows on."""
    dt = weight_dtype("uint4b")
    assert ops.plan(1, 7168, 2048, dt, 8, 128)["tile_m"] == 0 and ops.plan(M, 7168, 2048, dt, 8, 128)["tile_m"] == 16
    _forced(M, 7168, 2048, dt, 8, dict(), seed=M)
