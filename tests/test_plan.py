"""The plan table, without a GPU."""
import pytest
import torch

from tilus_b200 import _lib, ops


@pytest.fixture(scope="module", autouse=True)
def lib():
    from tilus_b200 import build

    build.build()
    return _lib.load()


def test_plans_are_reported_per_activation_type():
    """Up to 8 rows bfloat16 takes the stream kernel where fp16 takes the exact one; the plan says so, and asking for one
    type in between does not change what is reported for the other."""
    shape = (8, 6144, 4096, "uint4b", 8, 128)
    for _ in range(2):
        assert ops.plan(*shape)["tile_m"] == 16
        assert ops.plan(*shape, act_dtype=torch.bfloat16)["tile_m"] == 0
    assert ops.plan(9, *shape[1:], act_dtype=torch.bfloat16)["tile_m"] == 16
    for m in (1, 5, 8, 16, 100, 257, 300):  # one workspace serves both types
        both = [ops.plan(m, *shape[1:], act_dtype=t)["workspace_bytes"] for t in (torch.float16, torch.bfloat16)]
        assert ops.workspace_bytes(m, *shape[1:]) >= max(both)
    with pytest.raises(_lib.B200QError):
        ops.plan(8, 5120, 4100, "uint4b", 8, 128, act_dtype=torch.bfloat16)


@pytest.mark.parametrize("m,n,k,w,stream", [
    (4, 4096, 2048, "uint4b", True), (5, 4096, 4096, "uint4b", True), (8, 4096, 4096, "uint4b", True),
    (5, 28672, 4096, "uint4b", True), (8, 28672, 4096, "uint4b", False), (8, 32768, 2048, "uint4b", True),
    (8, 8192, 2048, "uint4b", False), (5, 4096, 2048, "uint4b", False), (8, 2048, 4096, "uint4b", False),
    (8, 2048, 8192, "uint4b", True), (5, 6144, 4096, "uint4b", False), (5, 1024, 4096, "float8_e5m2", True),
    (5, 2048, 2048, "int7b", False), (6, 8192, 2048, "int8", False), (5, 8192, 4096, "int8", True),
    (8, 4096, 4096, "int8", False), (9, 4096, 4096, "uint4b", False)])
def test_five_to_eight_rows_take_the_kernel_measured_faster(m, n, k, w, stream):
    """Both sides of every line of the rule, at shapes that were timed (fp16, one scale per 128 rows)."""
    zp = 8 if w == "uint4b" else 0
    assert (ops.plan(m, n, k, w, zp, 128)["tile_m"] == 0) is stream


def _static_ws_refused(lib, m, n, k, wtype, zero_point=0, group=128, act=0):
    """Whether b200q_gemm_static_ws turns the problem down for its scratch.  (Null operands: a problem that passes
    this check is refused for them, or for want of a GPU, right behind it.)"""
    return lib.b200q_gemm_static_ws(None, k, None, None, None, n, m, n, k, wtype, zero_point, group, act, None) \
        == _lib.ST_WORKSPACE


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("m", [1, 4, 5, 8, 16])
def test_static_workspace_takes_the_decode_path_up_to_one_width(lib, m, act):
    """16 fp32 sums and a count per column fit the built-in scratch up to 130,544 columns, whichever kernel the rows
    take; beyond, the problem stays refused."""
    int4 = (1 << 16) | (4 << 8)
    for n in (129280, 130544):
        assert not _static_ws_refused(lib, m, n, 7168, int4, act=act)
    assert _static_ws_refused(lib, m, 130560, 7168, int4, act=act)


@pytest.mark.parametrize("m,n,k", [(300, 9472, 4096), (329, 9280, 6656), (326, 6000, 2048), (1399, 1488, 1920), (272, 8592, 7936)])
def test_static_workspace_takes_prefill_batches_that_256_row_tiles_fit(lib, m, n, k):
    """Tiles of 384 rows come with a K split or larger slabs than the built-in scratch holds; tiles of 256 do without."""
    uint4 = 4 << 8
    assert ops.plan(m, n, k, "uint4b", 8, 128)["workspace_bytes"] > lib.b200q_static_workspace_limit()
    assert not _static_ws_refused(lib, m, n, k, uint4, 8)


@pytest.mark.parametrize("m", [7, 8])
@pytest.mark.parametrize("n", [2048, 8192, 14336, 18944, 28672, 32768])
@pytest.mark.parametrize("w", ["uint4b", "int8", "uint2b"])
def test_seven_and_eight_rows_do_not_cut_short_layers(m, n, w):
    """2048 rows of weights are one chunk, whose sums stay in shared memory (28672 columns in two chunks: a fifth slower)."""
    pl = ops.plan(m, n, 2048, w, 1 << (int(w[4]) - 1) if w[0] == "u" else 0, 128, act_dtype=torch.bfloat16)
    assert (pl["tile_m"], pl["splits"]) == (0, 1)


@pytest.mark.parametrize("m,n,k,w,ctas,warps", [
    (1, 16384, 1024, "uint2b", 256, 8), (2, 16384, 1024, "uint4b", 256, 8), (4, 16384, 1024, "uint4b", 256, 8), (8, 16384, 512, "uint4b", 256, 8), (1, 12288, 2048, "uint2b", 256, 8),
    (1, 8192, 1024, "int8", 256, 8), (1, 12288, 1536, "int5b", 256, 8),  # two CTAs of 8 warps per SM
    (4, 1024, 1024, "uint4b", 64, 8), (3, 2048, 1024, "uint4b", 128, 8), (5, 8192, 512, "uint2b", 128, 8), (4, 8192, 1024, "uint2b", 128, 8),  # one, with little to stage
    (1, 16384, 2048, "int8", 147, 16), (4, 4096, 2048, "uint4b", 128, 16), (1, 5120, 4096, "int3b", 107, 16),  # beyond those lines
    (8, 1024, 1024, "uint2b", 64, 16), (1, 8192, 8192, "uint4b", 128, 16)])
def test_small_decode_launches_have_ctas_of_eight_warps(m, n, k, w, ctas, warps):
    """Both sides of each line of the two rules, at shapes that were timed."""
    pl = ops.plan(m, n, k, w, 1 << (int(w[4]) - 1) if w[0] == "u" else 0, 128, act_dtype=torch.bfloat16)
    assert (pl["tile_m"], pl["splits"], pl["ctas_per_split"], pl["warps"]) == (0, 1, ctas, warps)
    assert pl["smem_bytes"] <= (113 if ctas > 148 else 227) * 1024


@pytest.mark.parametrize("m,n,k,w,splits", [
    (4, 1024, 14336, "uint4b", (4, 7, 14)), (3, 1024, 13824, "int8", (3, 9)), (6, 3072, 9216, "uint4b", (3, 6)), (6, 1536, 7168, "int8", (7,)),
    (5, 2048, 14336, "uint4b", (4, 7)), (6, 8192, 8192, "uint4b", (2, 4)), (8, 4096, 4096, "uint4b", (4,)),
    (4, 4096, 4096, "uint4b", (1,)), (6, 28672, 4096, "uint4b", (1,)), (5, 16384, 8192, "uint4b", (1,)), (2, 8192, 8192, "uint4b", (1,)),
    (1, 1024, 14336, "uint4b", (1,))])
def test_k_chunks_of_two_to_eight_rows(m, n, k, w, splits):
    """Narrow layers with long rows are cut, which saves staging; wide ones are not.  Any of the numbers given is within 6 % of the
    best that was timed."""
    pl = ops.plan(m, n, k, w, 8 if w[0] == "u" else 0, 128, act_dtype=torch.bfloat16)
    assert pl["tile_m"] == 0 and pl["splits"] in splits, pl


@pytest.mark.parametrize("m,n,k,w,act,resident", [
    (1, 28672, 4096, "uint4b", 0, 1), (1, 4096, 5120, "uint4b", 0, 1), (1, 6144, 5120, "uint4b", 0, 1), (1, 8192, 6144, "uint4b", 0, 0), (1, 4096, 8192, "uint4b", 0, 1), (1, 6144, 8192, "uint4b", 0, 1),
    (1, 8192, 8192, "uint4b", 0, 2), (1, 8192, 6144, "uint4b", 0, 0), (1, 8192, 2048, "uint2b", 0, 1), (1, 11008, 2048, "uint2b", 0, 0), (1, 16384, 4096, "int3b", 0, 1), (1, 28672, 14336, "uint4b", 0, 0), (1, 8192, 14336, "int3b", 0, 0),
    (1, 28672, 6144, "int3b", 0, 0), (1, 4096, 14336, "uint4b", 0, 4), (1, 4096, 14336, "float6_e3m2", 0, 0), (1, 28672, 14336, "int8", 0, 4), (1, 8192, 11008, "uint4b", 0, 2),
    (2, 4096, 4608, "uint4b", 0, 1), (2, 6144, 4608, "uint4b", 0, 1), (2, 8192, 4608, "uint4b", 0, 0), (4, 8192, 5120, "uint4b", 0, 1), (4, 16384, 5120, "uint4b", 0, 0), (4, 8192, 14336, "float6_e3m2", 0, 0),
    (8, 28672, 4096, "uint4b", 0, 1), (8, 4096, 5120, "uint4b", 0, 2), (8, 4096, 5120, "int8", 0, 1), (8, 8192, 8192, "uint4b", 0, 2), (8, 4096, 14336, "float6_e3m2", 0, 4),
    (8, 16384, 14336, "float6_e3m2", 0, 0), (8, 1024, 4224, "int6b", 0, 1), (8, 16384, 14336, "uint4b", 0, 2),
    (9, 11008, 4096, "uint4b", 0, 1), (9, 16384, 4096, "uint4b", 0, 1), (9, 18432, 4096, "uint4b", 0, 0), (9, 12288, 4096, "float6_e3m2", 0, 0), (13, 4096, 4096, "uint4b", 0, 1), (13, 6144, 4096, "uint4b", 0, 0),
    (15, 4096, 4096, "uint4b", 0, 0), (12, 4096, 4096, "int8", 0, 1), (13, 4096, 4096, "int8", 0, 0), (16, 4096, 2048, "int8", 0, 1), (16, 4096, 4096, "float6_e3m2", 0, 1),
    (16, 2048, 4096, "uint4b", 0, 0), (16, 8192, 1024, "uint4b", 0, 0), (9, 5120, 1024, "uint4b", 0, 1), (9, 6144, 1024, "uint4b", 0, 0), (16, 5120, 1024, "uint4b", 0, 0), (16, 6144, 1536, "int3b", 0, 1),
    (13, 6144, 1920, "int8", 0, 1), (9, 8192, 1920, "uint4b", 0, 0), (9, 8192, 2176, "uint4b", 0, 1), (13, 6144, 2176, "int3b", 0, 0), (13, 2560, 2560, "int3b", 0, 0), (16, 4096, 8192, "uint4b", 0, 0), (17, 4096, 4096, "uint4b", 0, 0),
    (8, 4096, 4096, "uint4b", 1, 1), (9, 4096, 4096, "uint4b", 1, 0), (8, 4096, 4224, "uint4b", 1, 0)])
def test_calls_that_keep_their_activations_in_registers(m, n, k, w, act, resident):
    """Both sides of the lines of the rule, at shapes that were timed.  bfloat16 only where the stream kernel had it: the tcgen05
    kernels have bfloat16's range."""
    pl = ops.plan(m, n, k, w, 1 << (int(w[4]) - 1) if w[0] == "u" else 0, 128, act_dtype=(torch.float16, torch.bfloat16)[act])
    assert pl["resident"] == resident
