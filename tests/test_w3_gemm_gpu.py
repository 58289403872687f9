"""The many-row kernel at the edges of its tiles, against the dequantised weights in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,k,t,dtype,scale_dtype,add", (
    ((32,), 128, 1, torch.bfloat16, torch.float16, False),            # a quarter row tile, one group, one token
    ((160,), 640, 17, torch.float16, torch.float16, True),            # an odd group count, a partial second row tile
    ((256, 64, 64), 1152, 257, torch.bfloat16, torch.float16, True),  # stacked matrices, two token tiles, the second short
    ((8192,), 384, 600, torch.bfloat16, torch.bfloat16, False),       # more tiles than SMs: accumulator and rings change hands
    ((4096,), 4096, 333, torch.bfloat16, torch.float16, False),
    # tiles of 256 tokens, three stages beside four operand slots: the MMA's two barriers are of different rounds; SMs with several tiles
    ((12288, 12288), 1152, 500, torch.bfloat16, torch.float16, False),
    ((12288,), 1152, 250, torch.bfloat16, torch.float16, True),       # one such tile of an SM, ragged
    ((12288,), 1152, 192, torch.float16, torch.bfloat16, False),      # the largest tile whose rings go round together
))
def test_many_rows(widths, k, t, dtype, scale_dtype, add):
    from marlin_style_fluxbin_b200 import _native

    gen = torch.Generator(device="cuda").manual_seed(sum(widths) + k + t)
    layouts = [{"planes": torch.randint(0, 256, (k // 128, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8),
                "scales": (torch.rand(k // 128, o, device="cuda", generator=gen) * 0.015 + 0.005).to(scale_dtype),
                "zeros": torch.randint(0, 8, (k // 128, o), device="cuda", generator=gen, dtype=torch.uint8)} for o in widths]
    x = torch.randn(t, k, device="cuda", generator=gen).to(dtype)
    addend = torch.randn(t, sum(widths), device="cuda", generator=gen).to(dtype) if add else None
    out = torch.full((t, sum(widths)), float("nan"), device="cuda", dtype=dtype)
    _native.w3_gemm(x, layouts, out, addend)
    dense = torch.empty(sum(widths), k, device="cuda", dtype=dtype)
    begin = 0
    for layout, o in zip(layouts, widths):
        _native.w3_dequant([(layout, dense[begin:begin + o])], dtype)
        begin += o
    want = x.double() @ dense.double().t() + (0 if addend is None else addend.double())
    size = x.double().abs() @ dense.double().abs().t()
    # fp32 sums of k / 16 instructions, each within 2^-22 of the magnitudes (aligned and cut off), and one rounding of the result
    bound = (k // 16 + 1) * 2.0 ** -22 * size + 2.0 ** (-8 if dtype == torch.bfloat16 else -11) * want.abs() + 2.0 ** -24
    assert bool(((out.double() - want).abs() <= bound).all())
    again = torch.empty_like(out)
    _native.w3_gemm(x, layouts, again, addend)
    assert torch.equal(again, out)
    assert _native.status_word() == 0
