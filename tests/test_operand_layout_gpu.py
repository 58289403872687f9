"""Operands of the packed entry points that do not lie as the kernels read them: rows apart, columns of a wider output, another device."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layout(o, k, device="cuda"):
    gen = torch.Generator().manual_seed(o + k)
    return {"planes": torch.randint(0, 256, (k // 128, 3, o, 16), generator=gen, dtype=torch.uint8).to(device),
            "scales": (torch.rand(k // 128, o, generator=gen) * 0.015 + 0.005).half().to(device),
            "perm": torch.randperm(k, generator=gen).to(torch.int16).to(device)}


@pytest.mark.parametrize("rows,kernel", ((1, "lut"), (3, "lut"), (3, "mma"), (16, "mma")))
def test_strided_operands(rows, kernel):
    from marlin_style_fluxbin_b200.w3_lut_deployment import w3_lut_gemv_out

    layout, gen = _layout(64, 256), torch.Generator(device="cuda").manual_seed(rows)
    wide = torch.randn(rows, 2 * 256 + 8, device="cuda", generator=gen).bfloat16()
    x = wide[:, 8:264]
    want = torch.empty(rows, 64, device="cuda", dtype=torch.bfloat16)
    w3_lut_gemv_out(x.contiguous(), layout, want, kernel=kernel)
    for strided in (x, x.t().contiguous().t()):
        for _ in range(3):  # plain, preparing, prepared
            around = torch.full((rows, 80), 7.0, device="cuda", dtype=torch.bfloat16)
            got = w3_lut_gemv_out(strided, layout, around[:, 8:72], kernel=kernel)
            assert torch.equal(got, want) and bool((around[:, :8] == 7).all()) and bool((around[:, 72:] == 7).all())


def test_one_row_entry_point_with_a_strided_row():
    from marlin_style_fluxbin_b200.w3_lut_deployment import w3_lut_m1_out, workspace_shape

    layout = _layout(64, 256)
    wide = torch.randn(1, 512, device="cuda").bfloat16()
    want, got, workspace = (torch.empty(shape, device="cuda", dtype=dtype) for shape, dtype in
                            (((1, 64), torch.bfloat16), ((1, 64), torch.bfloat16), (workspace_shape(64, 256), torch.float32)))
    w3_lut_m1_out(wide[:, ::2].contiguous(), layout, want, workspace, row_tile=256)
    w3_lut_m1_out(wide[:, ::2], layout, got, workspace, row_tile=256)
    assert torch.equal(got, want)


def test_weights_elsewhere_are_refused():
    from marlin_style_fluxbin_b200.w3_lut_deployment import w3_lut_gemv_out

    x, out = torch.zeros(2, 256, device="cuda", dtype=torch.bfloat16), torch.zeros(2, 64, device="cuda", dtype=torch.bfloat16)
    for _ in range(3):
        with pytest.raises(ValueError, match="device"):
            w3_lut_gemv_out(x, _layout(64, 256, "cpu"), out)
        with pytest.raises(ValueError, match="device"):
            w3_lut_gemv_out(x.cpu(), _layout(64, 256), out.cpu())
