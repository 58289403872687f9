"""Kernels of a prompt that are launched programmatically: SwiGLU rows over their chunks of a row, and that each waits for a launch
directly ahead which releases its dependents before it writes."""
import pytest
import torch

from marlin_style_fluxbin_b200 import _native

pytestmark = pytest.mark.gpu


def _check_gate(gate_up, out):
    width = out.shape[1]
    want = torch.nn.functional.silu(gate_up[:, :width].float()).to(out.dtype).float() * gate_up[:, width:].float()
    # the gate may round to its neighbour (exp is approximate), the product once more: two units in the last place of 8 or 11 bits, and of fp16's smallest
    ulp = 2.0 ** -7 if out.dtype == torch.bfloat16 else 2.0 ** -10
    floor = 0.0 if out.dtype == torch.bfloat16 else 2.0 ** -24
    assert bool(((out.float() - want).abs() <= 2 * ulp * want.abs() + 2 * floor * (1 + gate_up[:, width:].float().abs())).all())


@pytest.mark.parametrize("width", (8, 248, 2048, 2056, 2176, 4104, 12288, 25600))
@pytest.mark.parametrize("rows", (1, 5))
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
def test_gate_of_rows(width, rows, dtype):
    gen = torch.Generator(device="cuda").manual_seed(width + rows)
    gate_up = (torch.randn(rows, 2 * width, device="cuda", generator=gen) * 3).to(dtype)
    whole = torch.full((rows, width + 24), 7.0, device="cuda", dtype=dtype)
    out = whole[:, 8:8 + width]
    _native.silu_mul_rows(gate_up, out)
    _check_gate(gate_up, out)
    assert bool((whole[:, :8] == 7).all()) and bool((whole[:, 8 + width:] == 7).all())


def test_gate_of_a_row_of_more_chunks_than_a_grid_has():
    width = 65535 * 256 * 8 + 4104
    gate_up = torch.empty(1, 2 * width, device="cuda", dtype=torch.bfloat16).normal_(generator=torch.Generator(device="cuda").manual_seed(1))
    out = torch.full((1, width), float("nan"), device="cuda", dtype=torch.bfloat16)
    _native.silu_mul_rows(gate_up, out)
    _check_gate(gate_up, out)


@pytest.mark.parametrize("what", ("gate", "order", "heads"))
def test_what_the_launch_directly_ahead_writes(what):
    """The input is a one-row GEMV's output, in one graph; against the same call on what lies there when all is done."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    n, k = 6144, 255 * 128
    layout = (torch.randint(0, 256, (k // 128, 3, n, 16), device="cuda", generator=gen, dtype=torch.uint8), (torch.rand(k // 128, n, device="cuda", generator=gen) * 1e-3).bfloat16())
    xs = [torch.randn(1, k, device="cuda", generator=gen).bfloat16() for _ in range(2)]
    written, spare = (torch.zeros(1, n, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    normal = lambda *size: torch.randn(*size, device="cuda", generator=gen).bfloat16()  # noqa: E731
    perm, weights = torch.randperm(n, device="cuda", generator=gen).to(torch.int16), [normal(128) for _ in range(4)]
    outs = [torch.zeros(1, 32, 128, device="cuda", dtype=torch.bfloat16)] + [torch.zeros(8, 4, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    outs = {"gate": [torch.zeros(1, n // 2, device="cuda", dtype=torch.bfloat16)], "order": [torch.zeros(1, n, device="cuda", dtype=torch.bfloat16)], "heads": outs}[what]

    def call():
        if what == "gate":
            _native.silu_mul_rows(written, outs[0])
        elif what == "order":
            _native.gather_columns(written, perm, outs[0])
        else:
            _native.qknorm_rope_prompt(written, weights[0], weights[1], weights[2].view(1, 128), weights[3].view(1, 128), *outs, 1e-6)

    def body():
        _native.w3_gemv(xs[0], *layout, None, None, spare)
        _native.w3_gemv(xs[1], *layout, None, None, written)
        call()

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        body()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            body()
    for _ in range(5):
        torch.cuda.synchronize()
        written.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = [out.clone() for out in outs]
        call()
        torch.cuda.synchronize()
        assert all(bool(out.any()) and torch.equal(a, out) for a, out in zip(got, outs))
