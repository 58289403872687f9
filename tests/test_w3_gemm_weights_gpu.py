"""Weights of the many-row kernel read out one by one, in every pair of dtypes: with the identity as activations an output IS a weight (scales
from 1e-30 to where a weight overflows, zero points on either side of what the short forms cover); with a single weight that is not zero in
a row, every finite scale of 16 bits, where weights are subnormal or infinite too."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zero_points", ("none", "3 and 4", "any"))
@pytest.mark.parametrize("act_dtype", (torch.bfloat16, torch.float16))
@pytest.mark.parametrize("scale_dtype", (torch.bfloat16, torch.float16))
def test_every_scale(scale_dtype, act_dtype, zero_points):
    from marlin_style_fluxbin_b200 import _native

    k, o = 128, 65536
    gen = torch.Generator(device="cuda").manual_seed(7)
    scales = torch.arange(o, device="cuda", dtype=torch.int32).to(torch.int16).view(scale_dtype).clone()
    if zero_points == "any":  # short and long forms in one warp
        zeros = torch.randint(0, 256, (1, o), device="cuda", generator=gen, dtype=torch.uint8)
        zeros[:, ::3] = 4
    else:
        zeros = torch.randint(3, 5, (1, o), device="cuda", generator=gen, dtype=torch.uint8) if zero_points == "3 and 4" else torch.full((1, o), 4, device="cuda", dtype=torch.uint8)
    # what is not finite, or gives weights that are not, would meet a zero activation: out of the question here
    limit = 65504.0 / 256 if zero_points == "any" else 65504.0 / 4
    wide = scales.float().abs()
    if torch.float16 not in (scale_dtype, act_dtype):
        limit = 1e36
    scales = torch.where((wide <= limit) & ((wide >= 1e-30) | (wide == 0)), scales, torch.ones_like(scales))  # no fp32 subnormals
    planes = torch.randint(0, 256, (1, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8)
    bits = (planes.unsqueeze(-1) >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1  # [1, 3, O, 16, 8]
    codes = (bits[0, 0] + 2 * bits[0, 1] + 4 * (1 - bits[0, 2])).reshape(o, k).float()
    weights = (scales.view(o, 1).float() * (codes - zeros.view(o, 1).float())).to(scale_dtype).to(act_dtype)
    layout = {"planes": planes, "scales": scales.view(1, o)}
    if zero_points != "none":
        layout["zeros"] = zeros
    out = torch.empty(k, o, device="cuda", dtype=act_dtype)
    _native.w3_gemm(torch.eye(k, device="cuda", dtype=act_dtype), (layout,), out)
    assert torch.equal(out.T.float(), weights.float())


@pytest.mark.parametrize("zero", (None, 3, 0, 7))
@pytest.mark.parametrize("act_dtype", (torch.bfloat16, torch.float16))
@pytest.mark.parametrize("scale_dtype", (torch.bfloat16, torch.float16))
def test_one_weight_of_every_finite_scale(scale_dtype, act_dtype, zero):
    from marlin_style_fluxbin_b200 import _native

    o, z = 65536, 4 if zero is None else zero
    scales = torch.arange(o, device="cuda", dtype=torch.int32).to(torch.int16).view(scale_dtype)
    scales = torch.where(scales.isfinite(), scales, torch.ones_like(scales)).view(1, o)
    out = torch.empty(1, o, device="cuda", dtype=act_dtype)
    for code in range(8):
        codes = torch.full((128,), z, device="cuda", dtype=torch.int32)
        codes[16 * code + 3] = code
        bits = torch.stack((codes & 1, codes >> 1 & 1, 1 - (codes >> 2 & 1)))  # the high plane is stored inverted
        row = (bits.view(3, 16, 8) << torch.arange(8, device="cuda")).sum(-1).to(torch.uint8)
        layout = {"planes": row.view(1, 3, 1, 16).expand(1, 3, o, 16).contiguous(), "scales": scales}
        if zero is not None:
            layout["zeros"] = torch.full((1, o), zero, device="cuda", dtype=torch.uint8)
        _native.w3_gemm(torch.ones(1, 128, device="cuda", dtype=act_dtype), (layout,), out)
        want = (scales.float() * (code - z)).to(scale_dtype).to(act_dtype)  # one factor of eight bits or eleven, one of three: exact in fp32
        assert torch.equal(out, want), code


@pytest.mark.parametrize("o,k,t", ((160, 256, 128), (24576, 256, 128), (24576, 384, 100), (24576, 128, 128), (12288, 640, 333), (256, 640, 129)))
def test_tiles_of_two_accumulators(o, k, t):
    """Up to 128 tokens two warps take the groups of a tile in turns: one group, two, odd numbers of them, CTAs with several tiles."""
    from marlin_style_fluxbin_b200 import _native

    gen = torch.Generator(device="cuda").manual_seed(o + k + t)
    layout = {"planes": torch.randint(0, 256, (k // 128, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8),
              "scales": (torch.rand(k // 128, o, device="cuda", generator=gen) * 0.015 + 0.005).bfloat16()}
    x, addend = (torch.randn(t, n, device="cuda", generator=gen).bfloat16() for n in (k, o))
    out = torch.full((t, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    _native.w3_gemm(x, (layout,), out, addend)
    dense = torch.empty(o, k, device="cuda", dtype=torch.bfloat16)
    _native.w3_dequant([(layout, dense)], torch.bfloat16)
    want = x.double() @ dense.double().t() + addend.double()
    # fp32 sums of k / 16 instructions, each within 2^-22 of the magnitudes, two of them added, and one rounding of the result
    bound = (k // 16 + 2) * 2.0 ** -22 * (x.double().abs() @ dense.double().abs().t()) + 2.0 ** -8 * want.abs() + 2.0 ** -24
    assert bool(((out.double() - want).abs() <= bound).all())
    again = torch.empty_like(out)
    _native.w3_gemm(x, (layout,), again, addend)
    assert torch.equal(again, out)
    assert _native.status_word() == 0
