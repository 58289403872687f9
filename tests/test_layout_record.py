"""What the packed calls remember of a layout holds only while the tensors are as they were checked."""
import copy
import io

import numpy as np
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
    assert again is not record


def test_values_at_a_known_address_are_checked_again():
    """Buffers exchanged for others over the same memory: address and version are those that were checked."""
    module = w3.PackedW3Linear(_layout(), fallback="dense", row_tile=256)
    values = np.full((2, 64), 3, dtype=np.uint8)
    module.zeros = torch.from_numpy(values)
    module._require_valid_values(module.layout())
    values[:] = 9
    module.zeros = torch.from_numpy(values)
    with pytest.raises(ValueError, match="zero points"):
        module._require_valid_values(module.layout())


def test_checked_modules_are_copied_and_saved():
    module = w3.PackedW3Linear(_layout(), fallback="dense", row_tile=256)
    module._require_valid_values(module.layout())
    twin = copy.deepcopy(module)
    assert torch.equal(twin.planes, module.planes)
    file = io.BytesIO()
    torch.save(module, file)
    file.seek(0)
    assert torch.equal(torch.load(file, weights_only=False).planes, module.planes)
