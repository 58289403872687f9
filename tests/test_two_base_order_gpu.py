"""Two-base GEMV: scales, residual and refinement tensors that the launch directly ahead writes, where that launch has released its
dependents before it wrote a thing (as the one-row W3 kernel does)."""
import pytest
import torch

from marlin_style_fluxbin_b200 import _native, binary_global
from marlin_style_fluxbin_b200.deployment import PackedHybridLinear
from test_deployment import make_global_case, make_payload

pytestmark = pytest.mark.gpu


def _written_directly_ahead(constant, call, out):
    """``constant`` becomes the output of a GEMV over 255 groups, in one graph with ``call`` behind it; against ``call`` on what lies there when all is done."""
    dtype = constant.dtype if constant.dtype in (torch.float16, torch.bfloat16) else torch.bfloat16
    flat = constant.view(-1).view(dtype).view(1, -1)
    n, k = flat.shape[1], 255 * 128
    assert n % 32 == 0 and n <= 65536
    gen = torch.Generator(device="cuda").manual_seed(n)
    planes = torch.randint(0, 256, (k // 128, 3, n, 16), device="cuda", generator=gen, dtype=torch.uint8)
    scales = (torch.rand(k // 128, n, device="cuda", generator=gen) * 1e-4).half()
    xs = [torch.randn(1, k, device="cuda", generator=gen).to(dtype) for _ in range(2)]
    spare = torch.empty_like(flat)

    def body():
        _native.w3_gemv(xs[0], planes, scales, None, None, spare)
        _native.w3_gemv(xs[1], planes, scales, None, None, flat)
        call(True)

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        body()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            body()
    torch.cuda.synchronize()
    for _ in range(5):
        flat.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = out.clone()
        call(False)
        torch.cuda.synchronize()
        assert bool(torch.isfinite(got).all()) and bool(flat.any()) and torch.equal(got, out)


@pytest.mark.parametrize("o,groups,salient", ((2048, 8, 32), (2048, 16, 32), (1024, 8, 5), (2560, 32, 16)))
@pytest.mark.parametrize("name", ("row_scales", "column_scales", "salient_values"))
def test_matrix_wide_scales(o, groups, salient, name):
    layout, _, x = make_global_case(o, groups * 128, seed=o, n_sal=salient)
    layout, x = {key: value.cuda() for key, value in layout.items()}, x.cuda()
    out = torch.empty(1, o, device="cuda", dtype=x.dtype)
    _written_directly_ahead(layout[name], lambda pdl: _native.bb_global_gemv(
        x, *(layout[key] for key in binary_global.LAYOUT_FIELDS), out, pdl=pdl), out)


@pytest.mark.parametrize("kernel", ("v5", "v5_p1024"))
@pytest.mark.parametrize("name", ("rows", "columns", "sparse_rows", "sparse_columns", "sparse_codes"))
def test_scales_per_group(kernel, name):
    o, groups = 2048, 8
    layout = PackedHybridLinear(make_payload(o, groups), kernel=kernel).cuda().layout()
    x = torch.randn(1, groups * 128, generator=torch.Generator().manual_seed(o)).bfloat16().cuda()
    out = torch.empty(1, o, device="cuda", dtype=x.dtype)
    _written_directly_ahead(layout[name], lambda pdl: _native.bb_gemv(x, layout, out, pdl=pdl), out)
