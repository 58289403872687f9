"""Launches that follow one another on the same activations overlap: only where nothing but the activations is shared."""
import ctypes

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


class _Recorded:
    """Calls on a stand-in for the library that notes scratch and flags and may run something in the middle of a launch."""

    def __init__(self):
        from marlin_style_fluxbin_b200 import _native

        self.seen, self.between = [], None
        function = ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_void_p] * 4, ctypes.c_size_t, ctypes.c_uint, ctypes.c_void_p)
        self.run = function(self._run)
        self.ahead, self.scratch = {}, {}
        device = torch.cuda.current_device()
        self.call = _native.calls().Call(ctypes.cast(self.run, ctypes.c_void_p).value, 0, 1, 640, 96, device, torch.bfloat16, 0, _native.FB_W3_SAME_INPUT, 1, 256,
                                         _native._W3_SLOTS, self.scratch, self.ahead, self._allocate, torch.cuda.is_current_stream_capturing, None)

    def _allocate(self, index, size, family):
        return self.scratch.setdefault((index, torch.cuda.current_stream().cuda_stream, family), torch.zeros(256, dtype=torch.uint8, device="cuda"))

    def _run(self, launch, x, out, scratch, size, flags, stream):
        self.seen.append((scratch, flags))
        between, self.between = self.between, None
        if between is not None:
            between()
        return 0


def test_a_launch_during_another_threads_launch_waits():
    """What a second thread does while the first has given up the interpreter lock, played from inside the first one's launch."""
    recorded = _Recorded()
    x = torch.zeros(1, 640, device="cuda", dtype=torch.bfloat16)
    outs = [torch.empty(1, 96, device="cuda", dtype=torch.bfloat16) for _ in range(5)]
    recorded.call.run(x, outs[0])
    recorded.between = lambda: recorded.call.run(x, outs[1])
    recorded.call.run(x, outs[2])  # follows the first; the one in its middle cannot know what it follows
    recorded.call.run(x, outs[3])  # nor can the next
    recorded.call.run(x, outs[4])
    scratches, flags = zip(*recorded.seen)
    assert [bool(f) for f in flags] == [False, True, False, False, True]
    assert scratches[2] != scratches[1] and scratches[4] != scratches[3]


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
def test_a_capture_and_eager_launches_do_not_follow_one_another():
    recorded = _Recorded()
    x = torch.zeros(1, 640, device="cuda", dtype=torch.bfloat16)
    outs = [torch.empty(1, 96, device="cuda", dtype=torch.bfloat16) for _ in range(6)]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        recorded.call.run(x, outs[0])
        recorded.call.run(x, outs[1])
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            recorded.call.run(x, outs[2])  # nothing is ahead of it in the graph
            recorded.call.run(x, outs[3])
        recorded.call.run(x, outs[4])  # the captured ones have not run
        recorded.call.run(x, outs[5])
    assert [bool(flags) for _, flags in recorded.seen] == [False, True] * 3
