"""Device-side quantize-and-pack at the edges of its paths, against the oracle's arithmetic."""
import numpy as np
import pytest
import torch

from oracle import quant_oracle as qo
from tilus_b200 import dtypes as D
from tilus_b200 import packing, quantize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [D.int2b, D.int3b, D.int4b, D.int7b, D.int8, D.float3_e1m1, D.float7_e3m3],
                         ids=lambda d: d.name)
@pytest.mark.parametrize("k,group", [(128, 64), (384, 96), (1152, 384), (4096, 4096)])
@pytest.mark.parametrize("aligned", [True, False])
def test_rounding_boundaries_groups_and_alignment(dt, k, group, aligned):
    """Weights that are exact multiples of half a scale step sit on the rounding boundaries, where the
    reciprocal estimate must hand over to the division; groups that lie inside a warp's lanes and groups
    that need the pass of their own; rows on 16-byte boundaries and off them."""
    n = 32
    gen = torch.Generator().manual_seed(k + group)
    step = float(dt.max_value) * 2
    w = torch.randint(-int(step), int(step) + 1, (n, k), generator=gen).float() * 0.5 * 2.0 ** -6
    w[:, ::group] = float(dt.max_value) * 2.0 ** -6  # every group's absmax: the scale is 2^-6 exactly
    w[::2] *= 1.0 + 2.0 ** -9                        # every other column next to the boundaries instead
    wd = w.to(torch.float16).cuda()
    if not aligned:
        wd = torch.cat([wd.new_zeros(2), wd.reshape(-1)])[2:].view(n, k)
        assert wd.data_ptr() % 16 == 4
    packed, scales = quantize.quantize_and_pack(wd, dt, group)
    torch.cuda.synchronize()
    codes_ref, scales_ref = qo.quantize_weight(w.to(torch.float16).float().numpy(), dt, group)
    np.testing.assert_array_equal(scales.cpu().numpy().view(np.uint16), scales_ref.view(np.uint16))
    assert torch.equal(packed.cpu(), packing.interleave(torch.from_numpy(codes_ref), dt))
