"""Tensors off the boundary that a kernel reads them at are refused on the host: on the device they would be a fault."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _off(tensor):
    """The same values, one element past where an allocation begins."""
    flat = torch.empty(tensor.numel() + 1, device=tensor.device, dtype=tensor.dtype)
    flat[1:] = tensor.reshape(-1)
    return flat[1:].view(tensor.shape)


def test_two_base_activations_and_column_scales():
    from marlin_style_fluxbin_b200 import _native
    from marlin_style_fluxbin_b200.deployment import PackedHybridLinear
    from test_deployment import make_payload

    module = PackedHybridLinear(make_payload(64, 2)).cuda()
    x, out = torch.randn(1, 256, device="cuda").bfloat16(), torch.empty(1, 64, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(_native.NativeError, match="aligned"):
        _native.bb_gemv(_off(x), module.layout(), out)
    codes = torch.zeros(2, 64, 2, 16, device="cuda", dtype=torch.uint8)
    rows, columns = torch.ones(2, 64, device="cuda").half(), torch.ones(2, 256, device="cuda").half()
    with pytest.raises(_native.NativeError, match="aligned"):
        _native.bb_global_gemv(_off(x), codes, rows, columns, None, None, out)
    with pytest.raises(_native.NativeError, match="aligned"):
        _native.bb_global_gemv(x, codes, rows, _off(columns), None, None, out)
    _native.bb_gemv(x, module.layout(), _off(out))  # an output may lie anywhere
    _native.bb_global_gemv(x, codes, rows, columns, None, None, out)
    torch.cuda.synchronize()


def test_prompt_norm_and_rotation():
    from marlin_style_fluxbin_b200 import _native

    new = lambda *size: torch.ones(*size, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    plain = {"qkv": new(3, 4 * 128), "q_weight": new(128), "k_weight": new(128), "cos": new(3, 128), "sin": new(3, 128), "q_out": new(3, 2, 128),
             "k_cache": new(1, 8, 128), "v_cache": new(1, 8, 128)}
    for name in plain:
        with pytest.raises(_native.NativeError, match="aligned"):
            _native.qknorm_rope_prompt(**{**plain, name: _off(plain[name])}, eps=1e-6)
    _native.qknorm_rope_prompt(**plain, eps=1e-6)
    torch.cuda.synchronize()
