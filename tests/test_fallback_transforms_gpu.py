"""The dense fallback under what torch wraps around tensor operations: kernels launched with addresses must not pass it by."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _module(o=2080, k=256, bias=None):
    from marlin_style_fluxbin_b200.w3_lut_deployment import PackedW3Linear

    gen = torch.Generator().manual_seed(o)
    layout = {"planes": torch.randint(0, 256, (k // 128, 3, o, 16), generator=gen, dtype=torch.uint8),
              "scales": (torch.rand(k // 128, o, generator=gen) * 0.015 + 0.005).bfloat16(), "perm": torch.randperm(k, generator=gen).to(torch.int16)}
    return PackedW3Linear(layout, bias=bias, fallback="dense", row_tile=256).cuda()


def _near(got, want):
    """Two bf16 results: half a unit in the last place each, at most 2^-7 of the largest."""
    return float((got.float() - want.float()).abs().max()) <= 2.0 ** -7 * float(want.float().abs().max())


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning", "ignore::DeprecationWarning")
@pytest.mark.parametrize("rows", (5, 20))
def test_transforms_see_the_product(rows):
    module, x = _module(), torch.randn(2, rows, 256, device="cuda").bfloat16()
    tangent = torch.randn_like(x)
    with torch.no_grad():
        want = torch.stack([module(part) for part in x])
        assert _near(torch.func.vmap(module)(x), want)
        slope = module(tangent)
        assert _near(torch.func.jvp(module, (x,), (tangent,))[1], slope)
        with torch.autograd.forward_ad.dual_level():
            dual = module(torch.autograd.forward_ad.make_dual(x, tangent))
            assert _near(torch.autograd.forward_ad.unpack_dual(dual).tangent, slope)
        traced = torch.jit.trace(module, x[:1], check_trace=False)
        assert _near(traced(x[1:]), want[1:])


@pytest.mark.parametrize("rows", (5, 20, 1100))
def test_a_bias_of_another_dtype_stays_refused(rows):
    module = _module(bias=torch.randn(2080))
    with torch.no_grad(), pytest.raises(RuntimeError):
        module(torch.randn(1, rows, 256, device="cuda").bfloat16())
