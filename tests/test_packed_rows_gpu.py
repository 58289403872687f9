"""The packed kernel for 1..16 rows at the edges of its plan, against the dequantised product in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight(planes, scales, zeros):
    g, _, o, _ = planes.shape
    bits = (planes.unsqueeze(-1) >> torch.arange(8, device=planes.device, dtype=torch.uint8)) & 1
    bits = bits.reshape(g, 3, o, 128).double()
    code = bits[:, 0] + 2 * bits[:, 1] + 4 * (1 - bits[:, 2])  # the high plane is stored inverted
    zero = 4.0 if zeros is None else zeros.double().unsqueeze(-1)
    return ((code - zero) * scales.double().unsqueeze(-1)).permute(1, 0, 2).reshape(o, g * 128)


@pytest.mark.parametrize("o,k,m,dtype,options", (
    (32, 128, 2, torch.bfloat16, ""),                    # one task: fifteen idle warps
    (96, 640, 9, torch.float16, "zeros perm shifted"),   # an odd group count, tensors off the 16-byte boundary
    (160, 2944, 16, torch.bfloat16, "zeros perm add"),   # uneven shares of K
    (64, 32640, 16, torch.bfloat16, "zeros"),            # the largest K: eight rows per launch
    (65536, 4096, 16, torch.bfloat16, "zeros shifted"),  # the largest O: several batches of units
    (64, 512, 4, torch.bfloat16, "wild"),                # activations that dwarf their group, or are not finite
))
def test_packed_rows(o, k, m, dtype, options):
    from marlin_style_fluxbin_b200 import _native

    gen = torch.Generator(device="cuda").manual_seed(o + k + m)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)
    shift = 1 if "shifted" in options else 0

    def placed(t):  # the same values, one element past a boundary where asked
        flat = torch.empty(t.numel() + shift, device="cuda", dtype=t.dtype)
        flat[shift:] = t.reshape(-1)
        return flat[shift:].view(t.shape)

    g = k // 128
    planes = torch.randint(0, 256, (g, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8)
    scales = placed((torch.rand(g, o, device="cuda", generator=gen) * 0.015 + 0.005).half())
    zeros = placed(torch.randint(0, 8, (g, o), device="cuda", generator=gen, dtype=torch.uint8)) if "zeros" in options else None
    perm = placed(torch.randperm(k, device="cuda", generator=gen).to(torch.int16)) if "perm" in options else None
    x = (rand(m, k) * torch.exp2(4 * rand(m, k))).to(dtype)
    if "wild" in options:
        x[0, 7], x[1, 130], x[2, 300] = 1e30, float("inf"), 3e4
    addend = rand(m, o).to(dtype) if "add" in options else None
    out = torch.full((m, o), float("nan"), device="cuda", dtype=dtype)
    _native.w3_gemm_small(x, planes, scales, zeros, perm, out, addend=addend)
    weight = _weight(planes, scales, zeros)
    ordered = x.double() if perm is None else x.double()[:, perm.long()]
    finite = torch.isfinite(ordered)
    want = torch.where(finite, ordered, 0.0) @ weight.t()
    # fp32: eleven additions inside a group, one per group and per partial sum, each within 2^-23 of the sum of magnitudes
    size = torch.where(finite, ordered, 0.0).abs() @ (7 * scales.double()).t().repeat_interleave(128, dim=1).t()
    bound = (11 + g + 32) * 2.0 ** -23 * size
    if addend is not None:
        want += addend.double()
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -10)  # one ulp of the result
    error = (out.double() - want).abs()
    for row in range(m):
        if bool(finite[row].all()):
            assert bool((error[row] <= bound[row] + unit * want[row].abs() + 2.0 ** -24).all()), row
        else:  # an infinity reaches the outputs whose code is not zero, and leaves the others alone
            touched = weight[:, ~finite[row]].abs().sum(1) != 0
            assert bool((~torch.isfinite(out[row][touched])).all())
            assert bool((error[row][~touched] <= (bound[row] + unit * want[row].abs())[~touched]).all())
    for row in {0, m - 1}:  # whatever the other rows, and the number of them
        alone = torch.empty(1, o, device="cuda", dtype=dtype)
        _native.w3_gemm_small(x[row:row + 1].contiguous(), planes, scales, zeros, perm, alone, addend=None if addend is None else addend[row:row + 1].contiguous())
        assert torch.equal(alone[0].nan_to_num(), out[row].nan_to_num())


@pytest.mark.parametrize("top", (3e4, 3e9, 1e17, 1e30))
@pytest.mark.parametrize("m", (1, 4, 16))
def test_one_activation_above_all_others_of_its_group(m, top):
    """An output whose code is zero there sees the others alone, with the error that THEY give rise to: fp32 sums of three groups
    (the bound of the test above over the products that occur), one rounding, and nothing from the large one."""
    from marlin_style_fluxbin_b200 import _native

    gen = torch.Generator(device="cuda").manual_seed(m)
    o, k = 64, 384
    planes = torch.randint(0, 256, (3, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8)
    planes[0, :, :16, 77 // 8] &= 0xFF ^ 1 << 77 % 8  # code 4, the zero point, for sixteen outputs
    planes[1, :, :16, 72 // 8] &= 0xFF ^ 1 << 72 % 8
    scales = (torch.rand(3, o, device="cuda", generator=gen) * 0.015 + 0.005).half()
    x = torch.randn(m, k, device="cuda", generator=gen).bfloat16()
    x[:, 77], x[:, 128:256] = top, 0.0
    x[:, 200] = -top  # alone in its group
    out = torch.full((m, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    _native.w3_gemm_small(x, planes, scales, None, None, out)
    weight = _weight(planes, scales, None)
    want, size = x.double() @ weight.t(), x.double().abs() @ weight.abs().t()
    assert bool((size[:, :16] < 1e3).all())
    assert bool(((out.double() - want).abs() <= (11 + 3 + 32) * 2.0 ** -23 * size + 2.0 ** -8 * want.abs() + 2.0 ** -24).all())


@pytest.mark.parametrize("values", ((1e19, -3e19), (2.0 ** 127, 2.0 ** 126, 1e38), (-3.3895313892515355e38,), (-3.3895313892515355e38, -3.3895313892515355e38)))
@pytest.mark.parametrize("m", (1, 3, 16))
def test_finite_activations_up_to_the_largest(m, values):
    """Finite in, finite out: products with weights below one fit fp32 (the type's lowest value, as masks hold it, among them).  Several
    large ones share a group's scale, so what their own code hides is rounded with them: the bound of ``test_packed_rows``."""
    from marlin_style_fluxbin_b200 import _native

    gen = torch.Generator(device="cuda").manual_seed(m)
    o, k = 64, 384
    planes = torch.randint(0, 256, (3, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8)
    scales = (torch.rand(3, o, device="cuda", generator=gen) * 0.015 + 0.005).half()
    x = torch.randn(m, k, device="cuda", generator=gen).bfloat16()
    for at, value in zip((131, 140, 250), values):
        x[m - 1, at] = value
    out = torch.full((m, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    _native.w3_gemm_small(x, planes, scales, None, None, out)
    weight = _weight(planes, scales, None)
    want, size = x.double() @ weight.t(), x.double().abs() @ (7 * scales.double()).t().repeat_interleave(128, dim=1).t()
    assert bool(torch.isfinite(out).all())
    assert bool(((out.double() - want).abs() <= (11 + 3 + 32) * 2.0 ** -23 * size + 2.0 ** -8 * want.abs() + 2.0 ** -24).all())
