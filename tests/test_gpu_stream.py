"""The decode kernel where its split of the work and its rings can go wrong."""
import pytest
import torch

from tilus_b200 import dtypes as D
from tilus_b200 import ops

from .launches import kernels

pytestmark = pytest.mark.gpu


def _problem(M, N, K, dt, group=128, seed=0):
    """A problem that the decode kernel takes: with fp16 activations, or with bfloat16 where fp16 goes to the exact kernel.  The
    bfloat16 scales are fp16 numbers too, so that the reference's weights are rounded to fp16 in either case."""
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(seed)
    zp = 1 << (dt.nbits - 1) if dt.kind == D.KIND_UINT else 0
    act = next((t for t in (torch.float16, torch.bfloat16) if ops.plan(min(M, 16), N, K, dt, zp, group, act_dtype=t)["tile_m"] == 0),
               torch.float16)
    bq = torch.randint(0, 256, (N * K * dt.nbits // 8,), dtype=torch.uint8, device=dev, generator=gen)
    sc = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).to(act)
    a = torch.randn(M, K, device=dev, generator=gen).to(act)
    ref = a.float() @ ops.dequantize(bq, sc.half(), dt, group, zp).float()
    return a, bq, sc, zp, ref


def _close(c, ref):
    """One rounding of the output (2^-11 of it, bfloat16 2^-9) and one of each reference weight (2^-11)."""
    return float((c.float() - ref).abs().max()) <= (2e-3 if c.dtype == torch.float16 else 4e-3) * float(ref.abs().max())


def _run(a, bq, sc, dt, zp, ws=None):
    """The call on the decode kernel, as host-buffer and gather calls have it; others of most shapes go to the kernel that keeps the
    activations in registers."""
    return ops.quantized_matmul(a, bq, sc, dt, 128, zp, workspace=ws, plan_override=dict(resident=0))


@pytest.mark.parametrize("dt", [D.uint8, D.int8, D.uint7b, D.uint6b, D.int5b, D.uint4b, D.int3b, D.uint2b, D.uint1b, D.float6_e3m2],
                         ids=lambda d: d.name)
@pytest.mark.parametrize("M", [1, 2, 8])
def test_repeated_calls_with_the_weights_in_l2(dt, M):
    """A ring slot is refilled soonest when the copy finds its data in L2: every call of a warm series is right (8-bit
    types used to be read behind the refill where registers let the compiler delay their second loads)."""
    N, K = 2048, 8192
    a, bq, sc, zp, ref = _problem(M, N, K, dt)
    outs = [_run(a, bq, sc, dt, zp) for _ in range(40)]
    for c in outs:
        assert _close(c, ref)
    assert kernels(lambda: _run(a, bq, sc, dt, zp)) == ["stream_kernel"]


@pytest.mark.parametrize("M,N,K,dt", [
    (1, 2384, 1024, D.int8),      # 149 column tiles, two CTAs on one SM
    (1, 2384, 4096, D.int8),      # two tiles per CTA, the last CTA one
    (1, 5120, 1536, D.int3b),     # 107 CTAs of three tiles, the last two
    (2, 11008, 1024, D.uint8),    # 138 CTAs of five, the last three
    (1, 16, 512, D.uint4b),       # one tile: one CTA, half the warps
    (1, 16384, 1024, D.uint2b),   # two CTAs of 8 warps per SM
    (3, 12112, 1024, D.int5b),    # 253 such CTAs of three tiles, the last one
    (2, 4736, 2048, D.uint4b),    # one tile for each of two CTAs on every SM
    (4, 1040, 1024, D.float6_e3m2),  # 8 warps for four rows
    (8, 8192, 512, D.uint2b),     # and for eight (bfloat16)
    (2, 2368, 1024, D.uint2b),    # one tile per SM
    (3, 2384, 1024, D.float4_e2m1),
    (4, 160000, 512, D.uint1b),   # more tiles than a CTA owns: the rest item by item
    (8, 4096, 4096, D.uint4b),    # chunks of K, sums in the scratch
    (8, 8192, 4096, D.int6b),     # the same, with fewer tiles for the last CTA of a chunk (bfloat16)
    (7, 28672, 2048, D.int8)], ids=str)
def test_splits_of_the_column_tiles(M, N, K, dt):
    a, bq, sc, zp, ref = _problem(M, N, K, dt, seed=N)
    ws = torch.zeros(max(ops.workspace_bytes(M, N, K, dt, zp, 128), 1 << 20), dtype=torch.uint8, device=a.device)
    for _ in range(2):
        c = _run(a, bq, sc, dt, zp, ws)
        assert _close(c, ref)
    assert int(ws.count_nonzero()) == 0
    assert kernels(lambda: _run(a, bq, sc, dt, zp, ws)) == ["stream_kernel"]


@pytest.mark.parametrize("M,N,K,dt,stages", [(1, 8192, 8192, D.uint4b, 6), (1, 8192, 8192, D.uint4b, 8), (8, 4096, 4096, D.int8, 8),
                                             (4, 4096, 14336, D.uint4b, 5), (16, 2048, 2048, D.int6b, 8), (20, 2048, 2048, D.int3b, 8)], ids=str)
def test_plans_edited_to_deeper_rings(M, N, K, dt, stages):
    """Up to eight slots per warp may be asked for; as many are used as the launch has room for."""
    a, bq, sc, zp, ref = _problem(M, N, K, dt, seed=stages)
    pl = ops.plan(min(M, 4), N, K, dt, zp, 128)
    assert pl["tile_m"] == 0 and pl["stages"] < stages
    ws = torch.zeros(ops.workspace_bytes(16, N, K, dt, zp, 128), dtype=torch.uint8, device=a.device)
    call = lambda: ops.quantized_matmul(a, bq, sc, dt, 128, zp, workspace=ws, plan_override={**pl, "stages": stages})  # noqa: E731
    assert _close(call(), ref)
    assert set(kernels(call)) == {"stream_kernel"}
    assert int(ws.count_nonzero()) == 0
