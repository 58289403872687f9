"""Two-base GEMV at the edges of its units (32 rows), K blocks (one or two groups) and rings, against fp64."""
import pytest
import torch

from marlin_style_fluxbin_b200 import _native, binary_global
from marlin_style_fluxbin_b200.deployment import PackedHybridLinear, convert_artifact, decode_layout
from test_deployment import make_global_case, make_payload

pytestmark = pytest.mark.gpu


def _check(got, x, dense, groups):
    """One rounding to 16 bits (doubled), fp32 sums of at most 256 terms a chain (2^-24 each, so 2^-16 of the magnitudes; doubled), and
    the combine's fixed-point steps of 2^-26."""
    want, magnitude = x.double() @ dense.T, x.double().abs() @ dense.abs().T
    step = 2.0 ** -8 if x.dtype == torch.bfloat16 else 2.0 ** -11
    bound = step * want.abs() + 2.0 ** -15 * magnitude + groups * 2.0 ** -26
    assert bool(torch.isfinite(got).all())
    assert bool(((got.double().cpu() - want).abs() <= bound).all())


@pytest.mark.parametrize("o,groups,salient", ((1, 1, 0), (31, 5, 9), (33, 2, 5), (1024, 7, 4), (4064, 3, 3), (4065, 2, 2), (4096, 1, 1), (4097, 3, 3), (4128, 3, 2),
                                              (4100, 2, 7), (12320, 3, 4)))
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
def test_matrix_wide_scales(o, groups, salient, dtype):
    layout, _, x = make_global_case(o, groups * 128, seed=o + groups, n_sal=salient)
    x = x.to(dtype)
    out = torch.full((1, o), float("nan"), device="cuda", dtype=dtype)
    binary_global.global_two_base_m1_out(x.cuda(), {name: value.cuda() for name, value in layout.items()}, out)
    _check(out, x, binary_global.materialize(layout, torch.float64), groups)


@pytest.mark.parametrize("kernel", ("v5", "v5_p1024"))
@pytest.mark.parametrize("o,groups", ((1, 1), (31, 5), (1024, 2), (4064, 3), (4065, 2), (4096, 1), (4097, 3), (12320, 3)))
def test_scales_per_group(o, groups, kernel):
    payload = make_payload(o, groups, seed=o)
    x = torch.randn(1, groups * 128, generator=torch.Generator().manual_seed(o)).bfloat16()
    out = torch.full((1, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    _native.bb_gemv(x.cuda(), PackedHybridLinear(payload, kernel=kernel).cuda().layout(), out)
    _check(out, x, decode_layout(convert_artifact(payload, kernel=kernel), torch.float32).double(), groups)


@pytest.mark.parametrize("o,groups,salient", ((33, 1, 256), (4099, 2, 255), (12320, 3, 32), (9600, 2, 5)))
def test_more_residual_columns_than_groups(o, groups, salient):
    layout, _, x = make_global_case(o, groups * 128, seed=o + groups, n_sal=min(salient, groups * 128))
    out = torch.full((1, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    binary_global.global_two_base_m1_out(x.cuda(), {name: value.cuda() for name, value in layout.items()}, out)
    _check(out, x, binary_global.materialize(layout, torch.float64), groups)
