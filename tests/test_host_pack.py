"""The native converter of raw GPTQ words against the tensor-op form of the same conversion, bit for bit."""
import pytest
import torch

from marlin_style_fluxbin_b200 import _native
from marlin_style_fluxbin_b200.gptq_deployment import (
    convert_gptq_w3_to_planar, planes_from_sorted_codes, unpack_gptq_w3_qweight, unpack_gptq_w3_qzeros,
)

# without the library the tensor form would be compared with itself
pytestmark = pytest.mark.skipif(not _native.LIBRARY.exists(), reason="not built")


@pytest.mark.parametrize("o,k,desc_act", ((32, 128, False), (96, 640, True), (160, 256, True), (2048, 1024, True)))
def test_native_conversion_equals_the_tensor_form(o, k, desc_act):
    """Column counts around the 64-column blocks and 16-column transposes, one group and several, one thread and many."""
    gen = torch.Generator().manual_seed(o + k)
    word = lambda *size: torch.randint(-2**31, 2**31, size, dtype=torch.int64, generator=gen).to(torch.int32)  # noqa: E731
    order = torch.randperm(k, generator=gen) if desc_act else torch.arange(k)
    raw = {"qweight": word(3 * k // 32, o), "qzeros": word(k // 128, 3 * o // 32), "scales": torch.rand(k // 128, o, generator=gen).half(),
           "g_idx": (order // 128).to(torch.int32)}
    layout = convert_gptq_w3_to_planar(raw, general=True)
    by_group = torch.argsort(raw["g_idx"], stable=True)
    assert torch.equal(layout["planes"], planes_from_sorted_codes(unpack_gptq_w3_qweight(raw["qweight"])[by_group]))
    assert torch.equal(layout["zeros"], unpack_gptq_w3_qzeros(raw["qzeros"], qzero_format=1))
    assert torch.equal(layout["perm"].long(), by_group)


def test_column_orders_beyond_int16_are_refused():
    groups, order = (torch.arange(65536) // 128).to(torch.int32), torch.zeros(65536, dtype=torch.int64)
    assert _native.library().fb_host_w3_order(groups.data_ptr(), 65536, order.data_ptr()) == -2  # FB_ELIMIT
    assert not bool(order.any())
    assert _native.library().fb_host_w3_order(groups.data_ptr(), 32640, order.data_ptr()) == 0
    assert torch.equal(order[:32640], torch.arange(32640))
