"""Prepared launches against the plain entry points: same bits, whatever the stream, the layout's lifetime or its column order."""
import gc

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layout(o, k, seed, perm):
    gen = torch.Generator().manual_seed(seed)
    return {"planes": torch.randint(0, 256, (k // 128, 3, o, 16), generator=gen, dtype=torch.uint8).cuda(),
            "scales": (torch.rand(k // 128, o, generator=gen) * 0.015 + 0.005).half().cuda(),
            "zeros": torch.randint(3, 5, (k // 128, o), generator=gen, dtype=torch.uint8).cuda(),
            "perm": (torch.randperm(k, generator=gen) if perm else torch.arange(k)).to(torch.int16).cuda()}


@pytest.mark.parametrize("rows,kernel,arithmetic", ((1, "lut", "structural"), (1, "lut", "decoded_bf16"), (3, "lut", "structural"), (4, "lut", "decoded_bf16"),
                                                    (2, "mma", "structural"), (16, "mma", "structural")))
@pytest.mark.parametrize("perm", (False, True))
def test_repeated_calls_on_a_layout(rows, kernel, arithmetic, perm):
    from marlin_style_fluxbin_b200 import _native, w3_lut_deployment as w3

    layout = _layout(96, 640, rows, perm)
    xs = [torch.randn(rows, 640, generator=torch.Generator().manual_seed(i)).bfloat16().cuda() for i in range(3)]
    side = torch.cuda.Stream()
    for x in xs:  # the first call is the plain one, the second prepares, the third runs prepared
        want, got, there = (torch.full((rows, 96), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(3))
        column_order = layout["perm"] if perm else None
        if kernel == "mma":
            _native.w3_gemm_small(x, layout["planes"], layout["scales"], layout["zeros"], column_order, want)
        else:
            _native.w3_gemv(x, layout["planes"], layout["scales"], layout["zeros"], column_order, want, decoded_bf16=arithmetic == "decoded_bf16")
        w3.w3_lut_gemv_out(x, layout, got, arithmetic=arithmetic, kernel=kernel)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            w3.w3_lut_gemv_out(x, layout, there, arithmetic=arithmetic, kernel=kernel)
        side.synchronize()
        assert torch.equal(got, want) and torch.equal(there, want)
    assert any(isinstance(launch, _native.Launch) for launch in w3._RECORDS[id(layout["planes"])].launches.values())
    if rows == 1 and kernel == "lut":  # another column order written into the same tensor
        layout["perm"].copy_(torch.randperm(640, generator=torch.Generator().manual_seed(9)).to(torch.int16))
        fresh = {name: value.clone() for name, value in layout.items()}
        got, want = torch.empty(1, 96, device="cuda", dtype=torch.bfloat16), torch.empty(1, 96, device="cuda", dtype=torch.bfloat16)
        w3.w3_lut_gemv_out(xs[0], layout, got, arithmetic=arithmetic)
        w3.w3_lut_gemv_out(xs[0], fresh, want, arithmetic=arithmetic)
        assert torch.equal(got, want)
    key = id(layout["planes"])
    del layout
    gc.collect()
    assert key not in w3._RECORDS  # nothing outlives the planes


@pytest.mark.parametrize("rows,kernel", ((1, "lut"), (2, "mma")))
@pytest.mark.parametrize("name", ("planes", "scales"))
def test_an_output_inside_the_weights_is_refused_every_time(rows, kernel, name):
    from marlin_style_fluxbin_b200 import _native, w3_lut_deployment as w3

    layout = _layout(96, 640, 3, False)
    before = {key: value.clone() for key, value in layout.items()}
    x = torch.zeros(rows, 640, device="cuda", dtype=torch.bfloat16)
    out = layout[name].view(torch.bfloat16).view(-1)[:rows * 96].view(rows, 96)
    for _ in range(4):
        with pytest.raises(_native.NativeError, match="overlaps"):
            w3.w3_lut_gemv_out(x, layout, out, kernel=kernel)
    assert all(torch.equal(layout[key], before[key]) for key in layout)


def test_an_output_inside_two_base_codes_is_refused():
    from marlin_style_fluxbin_b200 import _native
    from marlin_style_fluxbin_b200.deployment import PackedHybridLinear
    from test_deployment import make_payload

    module = PackedHybridLinear(make_payload(64, 2)).cuda()
    lay = module.layout()
    launch = _native.Launch("bb", torch.bfloat16, tuple(lay[n] for n in ("codes", "rows", "columns", "sparse_codes", "sparse_rows", "sparse_columns", "indices")),
                            64, 256)
    before = module.codes.clone()
    with pytest.raises(_native.NativeError, match="overlaps"):
        launch(torch.zeros(1, 256, device="cuda", dtype=torch.bfloat16), module.codes.view(torch.bfloat16).view(-1)[:64].view(1, 64))
    assert torch.equal(module.codes, before)
