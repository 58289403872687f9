"""Two-base GEMV at the edges of its units (32 rows), K blocks (one or two groups, by size) and rings, against fp64."""
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


@pytest.mark.parametrize("o,groups,used,term", ((3104, 32, 2, 6400), (3104, 32, 32, 6400), (4128, 32, 31, 8000), (4064, 96, 96, 8000), (800, 255, 255, 8000), (64, 2, 2, 8000)))
@pytest.mark.parametrize("mode", ("matrix", "planar", "interleaved"))
def test_terms_up_to_the_limit(o, groups, used, term, mode):
    """Terms below 8192 in every group add up, also where a contribution carries two groups: one input a group, all signs positive, and
    scales that make every product exact."""
    k = groups * 128
    x = torch.zeros(1, k, dtype=torch.bfloat16)
    x[0, :used * 128:128] = term / 128
    if mode == "matrix":
        layout = binary_global.make_layout(torch.ones(2, o, k, dtype=torch.int8), torch.full((2, o), 8.0), torch.full((2, k), 8.0), torch.empty(0), torch.empty(o, 0))
        call = lambda out: binary_global.global_two_base_m1_out(x.cuda(), {name: value.cuda() for name, value in layout.items()}, out)  # noqa: E731
    else:
        shape = (groups, o, 2, 16) if mode == "planar" else (groups, o, 32)
        layout = {"codes": torch.full(shape, 255, dtype=torch.uint8), "rows": torch.full((groups, o, 2), 8.0), "columns": torch.full((groups, 128, 2), 8.0),
                  "sparse_codes": torch.zeros((groups, o, 2, 1) if mode == "planar" else (groups, o, 2), dtype=torch.uint8), "sparse_rows": torch.zeros(groups, o, 2),
                  "sparse_columns": torch.zeros(groups, 8, 2), "indices": torch.arange(8, dtype=torch.int16).repeat(groups, 1)}
        call = lambda out: _native.bb_gemv(x.cuda(), {name: value.cuda() for name, value in layout.items()}, out)  # noqa: E731
    out = torch.full((1, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    call(out)
    assert bool((out == torch.tensor(float(used * term)).bfloat16().cuda()).all())


def _first_of_two_groups(groups, planar, matrix_wide):
    """The smallest number of rows whose contributions carry two groups; one unit less must carry one."""
    count = lambda o: _native.library().fb_bb_gemv_block_groups(o, groups * 128, planar, matrix_wide)  # noqa: E731
    low, high = 1, 65536  # one group / two
    assert (count(low), count(high)) == (1, 2)
    while high - low > 1:
        middle = (low + high) // 2
        low, high = (low, middle) if count(middle) == 2 else (middle, high)
    return high


@pytest.mark.parametrize("rows_more", (-1, 0, 18, 31))
@pytest.mark.parametrize("groups,salient", ((2, 0), (2, 1), (3, 2), (3, 3), (3, 32), (5, 5), (5, 32), (9, 20), (2, 255)))
def test_matrix_wide_scales_on_either_side_of_two_groups(groups, salient, rows_more):
    o, k = _first_of_two_groups(groups, 1, 1) + rows_more, groups * 128
    gen = torch.Generator(device="cuda").manual_seed(o + salient)
    scale = lambda n: (torch.randn(2, n, device="cuda", generator=gen) * 0.02).abs().half()  # noqa: E731
    layout = {"codes": torch.randint(0, 256, (groups, o, 2, 16), device="cuda", generator=gen, dtype=torch.uint8), "row_scales": scale(o), "column_scales": scale(k),
              "salient_indices": torch.randperm(k, device="cuda", generator=gen)[:salient].int(),
              "salient_values": (torch.randn(o, salient, device="cuda", generator=gen) * 0.05).bfloat16()}
    x = torch.randn(1, k, device="cuda", generator=gen).bfloat16()
    out = torch.full((1, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    binary_global.global_two_base_m1_out(x, layout, out)
    _check(out, x.cpu(), binary_global.materialize(layout, torch.float64).cpu(), groups)


@pytest.mark.parametrize("rows_more", (-1, 0, 18, 31))
@pytest.mark.parametrize("groups,planar", ((8, 1), (9, 1), (7, 0), (8, 0)))
def test_scales_per_group_on_either_side_of_two_groups(groups, planar, rows_more):
    o = _first_of_two_groups(groups, planar, 0) + rows_more
    gen = torch.Generator(device="cuda").manual_seed(o)
    normal = lambda *size: torch.randn(*size, device="cuda", generator=gen)  # noqa: E731
    code = lambda *size: torch.randint(0, 256, size, device="cuda", generator=gen, dtype=torch.uint8)  # noqa: E731
    layout = {"codes": code(groups, o, 2, 16) if planar else code(groups, o, 32), "rows": normal(groups, o, 2) * 0.1, "columns": normal(groups, 128, 2),
              "indices": normal(groups, 128).argsort(1)[:, :8].sort(1).values.to(torch.int16).contiguous(),
              "sparse_codes": code(groups, o, 2, 1) if planar else code(groups, o, 2), "sparse_rows": normal(groups, o, 2) * 0.07, "sparse_columns": normal(groups, 8, 2)}
    x = normal(1, groups * 128).bfloat16()
    out = torch.full((1, o), float("nan"), device="cuda", dtype=torch.bfloat16)
    _native.bb_gemv(x, layout, out)
    _check(out, x.cpu(), decode_layout(layout, torch.float32).double().cpu(), groups)
