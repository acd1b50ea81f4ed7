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


@pytest.mark.parametrize("dt", [D.float3_e1m1, D.float4_e2m1, D.float5_e2m2, D.float6_e3m2, D.float6_e2m3, D.float7_e3m3, D.float5_e1m3, D.float8_e5m2, D.int3b, D.uint5b],
                         ids=lambda d: d.name)
@pytest.mark.parametrize("wdtype", [torch.float16, torch.bfloat16, torch.float32], ids=["f16", "bf16", "f32"])
@pytest.mark.parametrize("xdtype,group", [(torch.float16, 128), (torch.bfloat16, 96)])
def test_quotients_next_to_every_rounding_boundary(dt, wdtype, xdtype, group):
    """Quotients at every tie of the type and the fp32 numbers next to it, below the smallest number, at zeros of both signs and beyond the
    largest number (the scale's own rounding); scales that are powers of two and scales that are not.  Bit for bit."""
    n, k = 48, 384
    top = float(dt.max_value)
    steps = 64 if dt.nbits > 4 else 16
    gen = torch.Generator().manual_seed(dt.nbits)
    tie = (torch.randint(0, 2 * steps, (n, k), generator=gen) * 2 + 1).float() / (4 * steps) * 2.0 ** torch.randint(-18, 1, (n, k), generator=gen).float()
    w = tie * top * torch.where(torch.rand(n, k, generator=gen) < 0.5, -1.0, 1.0)
    w *= 1.0 + torch.randint(-2, 3, (n, k), generator=gen).float() * 2.0 ** -23
    w[:, 5::7] *= 2.0 ** -30
    w[:, 3::group] = 0.0
    w[:, 4::group] = -0.0
    w[:, ::group] = top
    w *= torch.where(torch.arange(n) % 2 == 0, torch.tensor(2.0 ** -6), 0.013 + torch.rand(n, generator=gen)).view(n, 1)
    w[7] *= 0.0
    wd = w.to(wdtype)
    packed, scales = quantize.quantize_and_pack(wd.cuda(), dt, group, xdtype)
    torch.cuda.synchronize()
    codes, want = quantize.quantize_weight(wd, dt, group, xdtype)
    assert torch.equal(scales.cpu().view(torch.int16), want.view(torch.int16))
    assert torch.equal(packed.cpu(), packing.interleave(codes, dt))


def _moved(layer, how):
    from torch import nn

    if how == "bfloat16":
        layer.bfloat16()  # scales only: the packed bytes stay uint8
    elif how == "float32":
        layer.scales = nn.Parameter(layer.scales.data.float(), requires_grad=False)
    elif how == "strided":
        layer.scales = nn.Parameter(torch.zeros(*layer.scales.shape[::-1], dtype=torch.float16, device="cuda").t(),
                                    requires_grad=False)
    elif how == "unaligned":
        buf = torch.zeros(layer.quantized_weight.numel() + 4, dtype=torch.uint8, device="cuda")
        layer.quantized_weight = nn.Parameter(buf[4:], requires_grad=False)
    elif how == "scales on the host":
        layer.scales = nn.Parameter(layer.scales.data.cpu(), requires_grad=False)


@pytest.mark.parametrize("how", ["as built", "bfloat16", "float32", "strided", "unaligned", "scales on the host"])
def test_load_into_parameters_of_any_kind(how):
    """load_and_quantize writes straight into the parameters only where the kernel may; into all others it copies,
    with the conversion that assignment implies."""
    from tilus_b200 import QuantizedLinear

    n, k, group, dt = 96, 512, 128, D.int4b
    w = (torch.randn(n, k, generator=torch.Generator().manual_seed(2)) * 0.1).half()
    layer = QuantizedLinear("float16", dt, group, k, n).cuda()
    _moved(layer, how)
    kind = layer.scales.dtype
    layer.load_and_quantize(w)
    torch.cuda.synchronize()
    codes, scales = qo.quantize_weight(w.float().numpy(), dt, group)
    assert torch.equal(layer.quantized_weight.data.cpu(), packing.interleave(torch.from_numpy(codes), dt))
    assert layer.scales.dtype == kind
    want = torch.from_numpy(scales).reshape(layer.scales.shape)
    assert torch.equal(layer.scales.data.cpu(), want.to(kind))


def test_out_tensors_that_do_not_fit_are_refused():
    w = torch.randn(32, 256, device="cuda").half()
    bq, sc = quantize.quantize_and_pack(w, D.int4b, 128)
    for out in ((bq[1:], sc), (bq, sc.float()), (bq, sc.t()), (bq.cpu(), sc), (bq[:-16], sc)):
        with pytest.raises(ValueError):
            quantize.quantize_and_pack(w, D.int4b, 128, out=out)


@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("kind", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("group", [32, 128, 256])
def test_signed_codes_of_ordinary_and_special_weights(bits, kind, group):
    """Units that need no clamping and those that do: zeros, weights so small that the least scale takes them beyond the
    range, infinities and NaN, single outliers, against the definition on the same device (codes are whole numbers: equal)."""
    dt, n, k = getattr(D, f"int{bits}b" if bits < 8 else "int8"), 64, 512
    gen = torch.Generator(device="cuda").manual_seed(bits + group)
    w = torch.randn(n, k, device="cuda", generator=gen) * 0.02
    w[0], w[1], w[2] = 0.0, 3e-7, w[2] * 1e-5
    w[3, 7], w[4, 9], w[5, 11] = float("inf"), float("-inf"), float("nan")
    w[6, ::37] *= 300.0
    w = w.to(kind)
    packed, scales = quantize.quantize_and_pack(w, dt, group, torch.float16)
    lo, hi = -float(1 << (bits - 1)), float((1 << (bits - 1)) - 1)
    x = w.float().reshape(n, k // group, group)
    amax = torch.nan_to_num(x.abs(), nan=0.0, posinf=float("inf")).amax(2)
    s = (amax / hi if hi else amax / torch.zeros_like(amax))
    s = torch.where(s.isnan(), s.new_tensor(1e-6), s.clamp(min=1e-6)).half()
    assert torch.equal(scales.view(torch.int16), s.t().contiguous().view(torch.int16))
    q = x / s.float()[:, :, None]
    q = torch.where(q.isnan(), q.new_tensor(lo), q.clamp(lo, hi)).round().reshape(n, k)
    codes = (q.to(torch.int32) & ((1 << bits) - 1)).to(torch.uint8).t().contiguous()
    assert torch.equal(packed.cpu(), packing.interleave(codes.cpu(), dt))


@pytest.mark.parametrize("n,k", [(16, 128), (48, 128), (80, 384), (16, 640), (144, 1152)])
@pytest.mark.parametrize("dt", [D.int4b, D.uint3b, D.float6_e3m2], ids=lambda d: d.name)
def test_groups_that_do_not_fill_the_last_block(n, k, dt):
    """A block takes four 128-row groups, of several column tiles where their number is odd; the last block has fewer."""
    w = (torch.randn(n, k, generator=torch.Generator().manual_seed(n + k)) * 0.1).half()
    guard = torch.full((n * k * dt.nbits // 8 + 4096,), 0x5a, dtype=torch.uint8, device="cuda")
    scales = torch.empty(k // 128, n, dtype=torch.float16, device="cuda")
    packed, scales = quantize.quantize_and_pack(w.cuda(), dt, 128, out=(guard[: -4096], scales))
    codes_ref, scales_ref = qo.quantize_weight(w.float().numpy(), dt, 128)
    np.testing.assert_array_equal(scales.cpu().numpy().view(np.uint16), scales_ref.view(np.uint16))
    assert torch.equal(packed.cpu(), packing.interleave(torch.from_numpy(codes_ref), dt))
    assert bool((guard[-4096:] == 0x5a).all())


def test_short_rows_take_no_longer_than_long_ones():
    """The same weights as rows of 128 and of 512: all threads of a block have work in both (26 us; 31 with three quarters of
    each block idle)."""
    best = {}
    dt, count = D.float6_e3m2, 65536 * 128
    w = [(torch.randn(count, device="cuda") * 0.02).half() for _ in range(4)]
    outs = {k: (torch.empty(count * 6 // 8, dtype=torch.uint8, device="cuda"), torch.empty(k // 128, count // k, dtype=torch.float16, device="cuda"))
            for k in (128, 512)}
    for _ in range(6):
        for k, out in outs.items():
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(2_000_000)  # the launches queue up behind it
            e0.record()
            for i in range(24):
                quantize.quantize_and_pack(w[i % 4].view(-1, k), dt, 128, out=out)
            e1.record()
            torch.cuda.synchronize()
            best[k] = min(best.get(k, 1e9), e0.elapsed_time(e1))
    assert best[128] <= 1.1 * best[512], best
