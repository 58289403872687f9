"""The dequantised-weight arithmetic of the one- to four-row kernel against the rounded weights in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(o, k, rows, dtype, scale_dtype, perm, zeros):
    gen = torch.Generator(device="cuda").manual_seed(o + k + rows)
    groups = k // 128
    layout = {"planes": torch.randint(0, 256, (groups, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8),
              "scales": (torch.rand(groups, o, device="cuda", generator=gen) * 0.015 + 0.005).to(scale_dtype),
              "perm": (torch.randperm(k, device="cuda", generator=gen) if perm else torch.arange(k, device="cuda")).to(torch.int16)}
    zero = torch.full((groups, o), 4, device="cuda", dtype=torch.uint8)
    if zeros:
        layout["zeros"] = zero = torch.randint(3, 5, (groups, o), device="cuda", generator=gen, dtype=torch.uint8)
    bits = (layout["planes"].unsqueeze(-1) >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1  # [G, 3, O, 16, 8]
    codes = (bits[:, 0] + 2 * bits[:, 1] + 4 * (1 - bits[:, 2])).reshape(groups, o, 128).float()
    weight = (layout["scales"].float().unsqueeze(-1) * (codes - zero.float().unsqueeze(-1))).to(scale_dtype).double()
    return layout, weight.permute(1, 0, 2).reshape(o, k), torch.randn(rows, k, device="cuda", generator=gen).to(dtype)


@pytest.mark.parametrize("rows,perm", ((1, False), (1, True), (2, False), (3, False), (3, True), (4, False)))
@pytest.mark.parametrize("o,k,zeros", ((32, 128, True), (96, 640, True), (96, 640, False), (2336, 4224, True)))
@pytest.mark.parametrize("dtype,scale_dtype", ((torch.bfloat16, torch.float16), (torch.float16, torch.bfloat16)))
def test_rounded_weights(o, k, zeros, rows, perm, dtype, scale_dtype):
    from marlin_style_fluxbin_b200.w3_lut_deployment import w3_lut_gemv_out

    layout, weight, x = _case(o, k, rows, dtype, scale_dtype, perm, zeros)
    out = torch.full((rows, o), float("nan"), device="cuda", dtype=dtype)
    w3_lut_gemv_out(x, layout, out, arithmetic="decoded_bf16", kernel="lut")
    ordered = x.double()[:, layout["perm"].long()]
    want, size = ordered @ weight.T, ordered.abs() @ weight.abs().T
    # one rounding to 16 bits (doubled), fp32 sums of at most 256 terms a chain (2^-16 of the magnitudes), 16 roundings to steps of 2^-26
    bound = 2.0 ** (-8 if dtype == torch.bfloat16 else -11) * want.abs() + 2.0 ** -16 * size + 2.0 ** -22
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("rows", (1, 3))
def test_an_infinite_activation(rows):
    """One that meets a code at the zero point adds nothing to the dot product nor to its correction; one above it gives infinity."""
    from marlin_style_fluxbin_b200.w3_lut_deployment import w3_lut_gemv_out

    layout, weight, x = _case(96, 256, rows, torch.bfloat16, torch.float16, False, False)
    x[:, 37] = float("inf")
    out = torch.empty(rows, 96, device="cuda", dtype=torch.bfloat16)
    w3_lut_gemv_out(x, layout, out, arithmetic="decoded_bf16", kernel="lut")
    at = weight[:, 37]
    assert bool(torch.isfinite(out[:, at == 0]).all()) and bool((out[:, at > 0] == float("inf")).all()) and not bool(torch.isfinite(out[:, at < 0]).any())
