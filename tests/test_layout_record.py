"""What the packed calls remember of a layout holds only while the tensors are as they were checked."""
import pytest
import torch

from marlin_style_fluxbin_b200 import w3_lut_deployment as w3


def _layout():
    return {"planes": torch.zeros(2, 3, 64, 16, dtype=torch.uint8), "scales": torch.ones(2, 64).half(), "zeros": torch.full((2, 64), 3, dtype=torch.uint8),
            "perm": torch.arange(256, dtype=torch.int16)}


@pytest.mark.parametrize("change", (
    lambda lay: lay["scales"].t_(),                         # another shape at the same address
    lambda lay: lay["planes"].transpose_(0, 1),
    lambda lay: lay["planes"].resize_(1, 3, 64, 16),
    lambda lay: lay["zeros"].as_strided_((2, 64), (1, 2)),  # the same shape, no longer contiguous
    lambda lay: lay["perm"].resize_(128),
))
def test_a_reshaped_tensor_is_checked_again(change):
    layout = _layout()
    record = w3._layout_record(layout)
    assert w3._layout_record(layout) is record
    change(layout)
    with pytest.raises(ValueError):
        w3._layout_record(layout)


def test_another_dtype_at_the_same_place_is_checked_again():
    layout = _layout()
    record = w3._layout_record(layout)
    layout["scales"].data = layout["scales"].data.view(torch.bfloat16)
    again = w3._layout_record(layout)
    assert again is not record and again.seen[1][4] == torch.bfloat16
