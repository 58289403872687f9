"""Launches that follow one another on the same activations overlap: only where nothing but the activations is shared."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layout(seed, o=96, k=640):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return {"planes": torch.randint(0, 256, (k // 128, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8),
            "scales": (torch.rand(k // 128, o, device="cuda", generator=gen) * 0.015 + 0.005).half(), "perm": torch.arange(k, device="cuda", dtype=torch.int16)}


def _in_a_row():
    from marlin_style_fluxbin_b200 import _native

    assert len(_native._same_input) == 1
    return next(iter(_native._same_input.values()))[1]


@pytest.mark.parametrize("prepared", (False, True))
def test_a_second_launch_into_the_same_output_waits(prepared):
    from marlin_style_fluxbin_b200 import _native

    x = torch.randn(1, 640, device="cuda").bfloat16()
    both = [_layout(seed) for seed in (1, 2)]
    outs = [torch.empty(1, 96, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    if prepared:
        launches = [_native.Launch("w3", torch.bfloat16, (lay["planes"], lay["scales"], None, None), 96, 640) for lay in both]
        call = lambda which, out: launches[which](x, out)  # noqa: E731
    else:
        call = lambda which, out: _native.w3_gemv(x, both[which]["planes"], both[which]["scales"], None, None, out)  # noqa: E731
    torch.cuda.synchronize()
    rows = []
    _native._same_input.clear()
    for which, out in ((0, outs[0]), (1, outs[1]), (0, outs[2]), (1, outs[0]), (0, outs[0]), (1, outs[1]), (0, outs[0])):
        call(which, out)
        rows.append(_in_a_row())
    assert rows == [1, 2, 3, 1, 1, 2, 1]
    want = torch.empty_like(outs[0])
    _native._same_input.clear()
    call(0, want)
    assert torch.equal(outs[0], want)
