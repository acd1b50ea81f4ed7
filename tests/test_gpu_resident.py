"""The decode kernel with the activations in registers, where its split of the work can go wrong."""
import pytest
import torch

from tilus_b200 import _lib
from tilus_b200 import dtypes as D
from tilus_b200 import ops
from tilus_b200.variants import supported_weight_dtypes

from .launches import kernels, launches

pytestmark = pytest.mark.gpu


def _problem(M, N, K, dt, group, act=torch.float16, mean=0.0, seed=0):
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(seed)
    zp = 1 << (dt.nbits - 1) if dt.kind == D.KIND_UINT else 0
    bq = torch.randint(0, 256, (N * K * dt.nbits // 8,), dtype=torch.uint8, device=dev, generator=gen)
    if dt.is_float() and dt.exponent_nbits == 5:
        bq &= 0xBF  # no Inf / NaN patterns
    sc = (torch.rand(K // group, N, device=dev, generator=gen) * 0.01 + 0.005).to(act)
    a = (torch.randn(M, K, device=dev, generator=gen) + mean).to(act)
    values = ops.dequantize(bq, torch.ones(1, N, dtype=torch.float16, device=dev), dt, K, zp).double()  # exact in fp16
    ref = a.double() @ (values * sc.double().repeat_interleave(group, 0))
    return a, bq, sc, zp, ref


def _close(c, ref):
    """No weight is rounded: one rounding of the output (2^-11, bfloat16 2^-8) and the fp32 sums, whose terms are up to
    a hundred times the result where the activations have a mean (a few 2^-24 of them: 2e-5 of the largest result)."""
    eps = 2.0 ** -11 if c.dtype == torch.float16 else 2.0 ** -8
    return bool(((c.double() - ref).abs() <= eps * ref.abs() + 2e-5 * ref.abs().max()).all())


def _run(a, bq, sc, dt, zp, group, S, ws=None, out=None):
    call = lambda: ops.quantized_matmul(a, bq, sc, dt, group, zp, workspace=ws, plan_override=dict(resident=S), out=out)  # noqa: E731
    c = call()
    assert (kernels(call) == ["resident_kernel"]) is (S > 0)
    return c


def _check(M, N, K, dt, group, S, act=torch.float16, mean=0.0):
    a, bq, sc, zp, ref = _problem(M, N, K, dt, group, act, mean, seed=M + N)
    ws = torch.zeros(max(ops.workspace_bytes(M, N, K, dt, zp, group), 1 << 16), dtype=torch.uint8, device=a.device)
    c = _run(a, bq, sc, dt, zp, group, S, ws)
    assert _close(c, ref)
    assert torch.equal(_run(a, bq, sc, dt, zp, group, S, ws), c)  # the sums are added in order
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("dt", supported_weight_dtypes(), ids=lambda d: d.name)
@pytest.mark.parametrize("M,K,S", [(5, 1024, 1), (16, 1152, 1), (8, 7168, 1), (3, 2432, 4)])
def test_every_weight_type(dt, M, K, S):
    _check(M, 1040, K, dt, 128, S, mean=3.0 if M == 5 else 0.0)


@pytest.mark.parametrize("M,N,K,group,S", [
    (1, 16, 128, 128, 1),          # one group of one tile: one warp has work
    (2, 16, 512, 512, 4),          # a cluster with one group each
    (8, 32, 8192, 128, 1),         # four groups per warp
    (8, 2368, 4096, 4096, 1),      # a tile per SM, one scale per column
    (7, 2384, 5120, 128, 1),       # two tiles, the last CTA one; some warps with a third group
    (4, 28672, 1024, 256, 1),      # sets of warps that take turns with 13 tiles
    (1, 14336, 2048, 128, 1),      # two sets with four and three tiles
    (16, 6144, 4096, 128, 1),      # 16 rows, three tiles
    (9, 4112, 2048, 1024, 1),      # 9 rows, the last CTA with one tile
    (8, 2064, 2176, 128, 2),       # 8.5 groups per CTA
    (5, 4096, 1024, 128, 8),       # eight CTAs to a cluster, a group each
    (2, 80, 9216, 128, 3),         # clusters of three, five tiles in all
    (8, 4096, 14336, 128, 4),
    (6, 4096, 14336, 7168, 2),     # seven groups for two warps
    (8, 75776, 1024, 128, 1),      # 32 tiles per CTA
    (3, 16400, 11008, 128, 2),     # 86 groups
])
def test_splits(M, N, K, group, S):
    _check(M, N, K, D.uint4b, group, S)


@pytest.mark.parametrize("M,K,S", [(1, 4096, 1), (8, 2048, 1), (8, 8192, 2), (5, 6144, 1)])
def test_bfloat16(M, K, S):
    _check(M, 1040, K, D.int4b, 128, S, act=torch.bfloat16)


def test_bfloat16_out_of_range():
    """Magnitudes that fp16 does not have saturate (infinities too); NaN stays NaN."""
    a, bq, sc, zp, _ = _problem(4, 64, 1024, D.int4b, 128, torch.bfloat16)
    a[0, 5], a[1, 7], a[2, 9] = 1e6, float("inf"), float("nan")
    c = _run(a, bq, sc, D.int4b, zp, 128, 1)
    b = a.clone()
    b[0, 5] = b[1, 7] = 65504.0
    ref = b.double() @ ops.dequantize(bq, sc, D.int4b, 128, zp).double()
    assert float((c - ref)[[0, 1, 3]].abs().max() / ref[[0, 1, 3]].abs().max()) <= 2.0 ** -7
    assert bool(c[2].isnan().all())


@pytest.mark.parametrize("scale", [2.0 ** -20, 2.0 ** -9, 400.0])
def test_activations_of_any_magnitude_are_multiplied_as_they_are(scale):
    """No power of two is taken off the activations beforehand: small fp16 values keep their bits."""
    a, bq, sc, zp, _ = _problem(3, 272, 2048, D.uint4b, 128)
    a = (a.float() * scale).half()
    sc = sc.float().div(scale if scale < 1 else 1).clamp(max=60000).half()
    values = ops.dequantize(bq, torch.ones(1, 272, dtype=torch.float16, device=a.device), D.uint4b, 2048, zp).double()
    ref = a.double() @ (values * sc.double().repeat_interleave(128, 0))
    assert _close(_run(a, bq, sc, D.uint4b, zp, 128, 1), ref)


@pytest.mark.parametrize("M,dt,mean", [
    (8, D.uint8, 3.0), (8, D.int8, 0.0), (16, D.int8, 3.0), (8, D.uint7b, 3.0), (16, D.int7b, 3.0), (8, D.int7b, 0.0), (4, D.uint5b, 0.0),
    (4, D.int6b, 0.0), (4, D.uint4b, 0.0), (8, D.int4b, 0.0), (8, D.uint3b, 0.0), (4, D.uint8, 3.0), (8, D.uint2b, 0.0)], ids=str)
def test_results_as_near_as_those_of_the_kernel_beside_it(M, dt, mean):
    """The share of results that are not the nearest fp16 value measures the error of the sums: 2^11 times that error.  Next to the
    stream (M <= 4) and exact kernels' on the same operands, plus four standard deviations of a count of that size."""
    N, K, group = 16384, 2048, 128
    a, bq, sc, zp, ref = _problem(M, N, K, dt, group, mean=mean, seed=3)
    nearest = ref.half()
    ws = torch.zeros(ops.workspace_bytes(M, N, K, dt, zp, group), dtype=torch.uint8, device=a.device)
    here, there = (int((_run(a, bq, sc, dt, zp, group, S, ws) != nearest).sum()) for S in (1, 0))
    assert here <= there + 4 * there ** 0.5


@pytest.mark.parametrize("M,gap", [(1, 1), (8, 3), (16, 8)])
def test_outputs_inside_a_wider_tensor(M, gap):
    a, bq, sc, zp, ref = _problem(M, 272, 1024, D.uint4b, 128)
    wide = torch.full((M, 272 + gap), 7.0, dtype=torch.float16, device=a.device)
    _run(a, bq, sc, D.uint4b, zp, 128, 1, out=wide[:, :272])
    assert _close(wide[:, :272], ref) and bool((wide[:, 272:] == 7.0).all())


def test_edits_of_other_fields_leave_the_kernel():
    a, bq, sc, zp, ref = _problem(8, 4096, 4096, D.uint4b, 128)
    pl = ops.plan(8, 4096, 4096, D.uint4b, zp, 128)
    assert pl["resident"] == 1
    run = lambda plan, x=a: ops.quantized_matmul(x, bq, sc, D.uint4b, 128, zp, plan_override=plan)  # noqa: E731
    c = run(None)
    assert torch.equal(run(pl), c)
    edits = {"stream_kernel": [dict(resident=0), dict(splits=2), dict(stages=pl["stages"] - 1), dict(ctas_per_split=100), dict(kernel=2, stages=2, ctas_per_split=100)],
             "exact_kernel": [dict(kernel=3, tile_m=16, splits=1, ctas_per_split=90), dict(tile_m=16, splits=1, ctas_per_split=90)]}
    for name, plans in edits.items():
        for plan in plans:
            assert float((run(plan).double() - ref).abs().max()) <= 2e-3 * float(ref.abs().max())
            assert kernels(lambda: run(plan)) == [name], plan
    rows = torch.randn(20, 4096, device=a.device).half()  # a plan put on more rows than the kernel takes
    got = run(pl, rows)
    want = rows.float() @ ops.dequantize(bq, sc, D.uint4b, 128, zp).float()
    assert float((got.float() - want).abs().max()) <= 2e-3 * float(want.abs().max())
    assert kernels(lambda: run(None), lambda: run(pl), lambda: run(pl, rows)) == ["resident_kernel", "resident_kernel", "stream_kernel", "stream_kernel"]


@pytest.mark.parametrize("M,K,ok", [(1, 1024, True), (8, 1024, True), (16, 1024, True), (1, 1152, False), (5, 1152, False), (16, 1152, False),
                                    (1, 4224, False), (8, 8320, False)])
@pytest.mark.parametrize("N", [272, 4112, 16384])
def test_rows_of_any_distance_do_not_depend_on_the_route(M, N, K, ok):
    """K in whole 512-row blocks takes outputs at any row stride, and asks for the stream kernel's scratch then; other K ask for multiples of
    eight elements, whichever kernel a width goes to."""
    a, bq, sc, zp, ref = _problem(M, N, K, D.uint4b, 128)
    wide = torch.zeros(M, N + 3, dtype=torch.float16, device=a.device)
    run = lambda ws=None, out=wide[:, :N]: ops.quantized_matmul(a, bq, sc, D.uint4b, 128, zp, out=out, workspace=ws)  # noqa: E731
    if ok:
        run()
        assert _close(wide[:, :N], ref)
        small = torch.zeros(256 + 4 * (N // 16 + 64) + 256, dtype=torch.uint8, device=a.device)
        with pytest.raises(_lib.B200QError):
            run(small)
    else:
        with pytest.raises(_lib.B200QError):
            run()
        assert int(wide.count_nonzero()) == 0
        run(out=torch.empty(M, N, dtype=torch.float16, device=a.device))


@pytest.mark.parametrize("M,N,K", [(8, 4096, 4096), (1, 8192, 8192), (16, 4096, 2048)])
def test_a_plan_says_whether_the_launch_overlaps_the_one_before(M, N, K):
    """pdl = 0 is for callers whose previous kernel writes weights or scales and releases its dependents early."""
    a, bq, sc, zp, ref = _problem(M, N, K, D.uint4b, 128)
    pl = ops.plan(M, N, K, D.uint4b, zp, 128)
    assert pl["resident"] > 0 and pl["pdl"] == 1
    early, late = (lambda pdl=pdl: ops.quantized_matmul(a, bq, sc, D.uint4b, 128, zp, plan_override=dict(pdl=pdl)) for pdl in (1, 0))
    assert _close(late(), ref) and torch.equal(early(), late())
    assert [e for _, e in launches(early, early, late, early, late)] == [False, True, False, True, False]
    assert set(kernels(early, late)) == {"resident_kernel"}


@pytest.mark.parametrize("M,N,K,dt", [
    (1, 2384, 1024, D.int8), (1, 5120, 1536, D.int3b), (2, 11008, 1024, D.uint8), (1, 16, 512, D.uint4b), (3, 12112, 1024, D.int5b),
    (4, 1040, 1024, D.float6_e3m2), (4, 160000, 512, D.uint1b), (8, 4096, 4096, D.uint4b), (1, 28672, 8192, D.uint4b),
    (8, 6144, 4096, D.uint4b), (16, 4096, 4096, D.int8), (12, 2064, 1152, D.uint2b), (5, 1040, 1408, D.float6_e3m2)], ids=str)
def test_the_kernels_beside_it(M, N, K, dt):
    """The stream and exact kernels at shapes that the table gives to this one: other callers (host buffers, gathers,
    edited plans) still have them."""
    a, bq, sc, zp, ref = _problem(M, N, K, dt, 128)
    ws = torch.zeros(max(ops.workspace_bytes(M, N, K, dt, zp, 128), 1 << 16), dtype=torch.uint8, device=a.device)
    for _ in range(2):
        assert _close(_run(a, bq, sc, dt, zp, 128, 0, ws), ref)
        assert int(ws.count_nonzero()) == 0
