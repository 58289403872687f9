"""Prompts that the kernels of the prompt path do not take run as tensor operations."""
import pytest
import torch


@pytest.mark.parametrize("dtype,head_dim", ((torch.float32, 128), (torch.float32, 64), (torch.bfloat16, 128)))
@pytest.mark.parametrize("device", ("cpu", pytest.param("cuda", marks=pytest.mark.gpu)))
def test_prefill_beyond_the_prompt_kernels(device, dtype, head_dim):
    """Devices, dtypes and head widths that the kernels do not take: against the fp32 yardstick of the same engine.  fp32: sums
    of at most 384 products, 2^-24 each, through two layers; bf16: a 16-bit pipeline of two layers."""
    from marlin_style_fluxbin_b200.decode_engine import DecodeEngine, ModelShape

    shape = ModelShape(layers=2, hidden=256, q_heads=4, kv_heads=2, head_dim=head_dim, intermediate=384, vocab=97)
    ids = torch.randint(0, 97, (1, 9), generator=torch.Generator().manual_seed(1))
    found = [DecodeEngine(shape, device=device, max_positions=16, dtype=dtype, arm=arm, seed=3) for arm in ("w3", "bf16")]
    logits = [engine.prefill(ids).float() for engine in found]
    truth = found[0].truth_logits(ids[:, :-1], ids[0, -1:])
    for got in logits:
        assert float((got - truth).norm() / truth.norm()) < (1e-4 if dtype == torch.float32 else 0.03)
    assert float(found[0].k_cache[:, :, :9].abs().amin(-1).max()) > 0 and float(found[0].k_cache[:, :, 9:].abs().max()) == 0
