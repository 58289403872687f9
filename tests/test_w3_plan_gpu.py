"""One-row GEMV around the line where a launch takes one CTA per SM instead of two, and the column order is read first."""
import pytest
import torch

from test_w3_lut_gpu import assert_parity, make_case, oracle_outputs, to_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,k", ((32, 128), (2304, 4096), (2336, 4096), (1152, 12288), (1184, 12288), (2336, 640)))
@pytest.mark.parametrize("perm", (False, True))
@pytest.mark.parametrize("rows", (1, 2))
def test_either_side_of_the_line(o, k, perm, rows):
    from marlin_style_fluxbin_b200.w3_lut_deployment import w3_lut_gemv_out

    layout, x = make_case(o, k, seed=o + k, perm=perm, zeros=not perm, m=rows)
    reference, _ = oracle_outputs(layout, x)
    out = torch.full((rows, o), float("nan"), device="cuda", dtype=x.dtype)
    w3_lut_gemv_out(x.cuda(), to_cuda(layout), out, kernel="lut")
    assert_parity(out, reference)
