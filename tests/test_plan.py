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
    shape = (8, 5120, 4096, "uint4b", 8, 128)
    for _ in range(2):
        assert ops.plan(*shape)["tile_m"] == 16
        assert ops.plan(*shape, act_dtype=torch.bfloat16)["tile_m"] == 0
    assert ops.plan(9, *shape[1:], act_dtype=torch.bfloat16)["tile_m"] == 16
    for m in (1, 5, 8, 16, 100, 257, 300):  # one workspace serves both types
        both = [ops.plan(m, *shape[1:], act_dtype=t)["workspace_bytes"] for t in (torch.float16, torch.bfloat16)]
        assert ops.workspace_bytes(m, *shape[1:]) >= max(both)
    with pytest.raises(_lib.B200QError):
        ops.plan(8, 5120, 4100, "uint4b", 8, 128, act_dtype=torch.bfloat16)
