"""Residual additions inside the bound W3 projections of a session's decode steps, against the stock modules."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shuffled", ((torch.bfloat16, True), (torch.float16, False)))
def test_steps_with_packed_projections(dtype, shuffled, monkeypatch):
    """NRMSE of the logits at the level of a 16-bit pipeline (two layers, 2^-8 per rounding for bf16)."""
    from transformers import Qwen3Config, Qwen3ForCausalLM

    from marlin_style_fluxbin_b200.fused_modules import fused_qwen3_modules
    from marlin_style_fluxbin_b200.qwen3 import QWEN3_LINEAR_MODULES
    from marlin_style_fluxbin_b200.static_decode import StaticDecodeSession, prepared_linears
    from marlin_style_fluxbin_b200.w3_lut_deployment import PackedW3Linear, replace_w3_block_linears

    torch.manual_seed(5)
    gen = torch.Generator(device="cuda").manual_seed(5)
    config = Qwen3Config(vocab_size=96, hidden_size=256, intermediate_size=384, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=128)
    config._attn_implementation = "sdpa"
    model = Qwen3ForCausalLM(config).eval().cuda().to(dtype)
    for block in model.model.layers:
        payload, tiles = {}, {}
        for name in QWEN3_LINEAR_MODULES:
            old = block.get_submodule(name)
            o, k = old.out_features, old.in_features
            payload[f"{name}.planes"] = torch.randint(0, 256, (k // 128, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8)
            payload[f"{name}.scales"] = (torch.rand(k // 128, o, device="cuda", generator=gen) * 0.015 + 0.005).bfloat16()
            payload[f"{name}.perm"] = (torch.randperm(k, device="cuda", generator=gen) if shuffled else torch.arange(k, device="cuda")).to(torch.int16)
            tiles[(o, k)] = 256
        replace_w3_block_linears(block, payload, fallback="dense", row_tile_by_shape=tiles)
    ids = torch.randint(0, 96, (1, 7), device="cuda", generator=gen)
    forced = torch.randint(0, 96, (1, 4), device="cuda", generator=gen)
    session = StaticDecodeSession(model, ids, forced)
    joined, plain = [], PackedW3Linear.add_to
    monkeypatch.setattr(PackedW3Linear, "add_to", lambda self, *a: (joined.append(1), plain(self, *a))[1])
    with prepared_linears(model, dtype):
        stock = session.audit()
        assert not joined
        with fused_qwen3_modules():
            fused = session.audit()
            assert len(joined) == 2 * 2 * 4  # two projections of two layers in four steps
            assert fused["routes"] == stock["routes"]
            graph = session.capture()
            assert torch.equal(graph["logits"], fused["logits"])
            joined.clear()
            handle = model.model.layers[0].mlp.register_forward_hook(lambda *a: None)
            session.audit()
            handle.remove()
            assert len(joined) == 2 * 4  # an observed MLP is called, not passed over
    gap = (fused["logits"].float() - stock["logits"].float()).square().mean().sqrt() / stock["logits"].float().square().mean().sqrt()
    assert float(gap) < 0.02


@pytest.mark.parametrize("change", ("attention", "mlp", "projection"))
def test_exchanged_parts_are_called(change):
    """A layer whose attention, MLP or projection has a forward of its own is not run past it; logits as by the stock layer."""
    from transformers import Qwen3Config, Qwen3ForCausalLM

    from marlin_style_fluxbin_b200.fused_modules import fused_qwen3_modules
    from marlin_style_fluxbin_b200.qwen3 import QWEN3_LINEAR_MODULES
    from marlin_style_fluxbin_b200.static_decode import StaticDecodeSession, prepared_linears
    from marlin_style_fluxbin_b200.w3_lut_deployment import PackedW3Linear

    torch.manual_seed(5)
    gen = torch.Generator(device="cuda").manual_seed(5)
    config = Qwen3Config(vocab_size=96, hidden_size=256, intermediate_size=384, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2, head_dim=128)
    config._attn_implementation = "sdpa"
    model = Qwen3ForCausalLM(config).eval().cuda().bfloat16()
    block = model.model.layers[0]
    for name in QWEN3_LINEAR_MODULES:
        old = block.get_submodule(name)
        o, k = old.out_features, old.in_features
        layout = {"planes": torch.randint(0, 256, (k // 128, 3, o, 16), device="cuda", generator=gen, dtype=torch.uint8),
                  "scales": (torch.rand(k // 128, o, device="cuda", generator=gen) * 0.015 + 0.005).bfloat16(),
                  "perm": torch.arange(k, device="cuda").to(torch.int16)}
        parent, attribute = name.rsplit(".", 1)
        setattr(block.get_submodule(parent), attribute, PackedW3Linear(layout, fallback="dense", row_tile=256))
    part = {"attention": block.self_attn, "mlp": block.mlp, "projection": block.mlp.down_proj}[change]

    def tripled(self, *args, **kwargs):
        out = super(part.__class__, self).forward(*args, **kwargs)
        return (out[0] * 3, *out[1:]) if isinstance(out, tuple) else out * 3

    part.__class__ = type("Own", (type(part),), {"forward": tripled})
    session = StaticDecodeSession(model, torch.randint(0, 96, (1, 7), device="cuda", generator=gen), torch.randint(0, 96, (1, 3), device="cuda", generator=gen))
    with prepared_linears(model, torch.bfloat16):
        stock = session.audit()["logits"].float()
        with fused_qwen3_modules():
            fused = session.audit()["logits"].float()
    assert float((fused - stock).square().mean().sqrt() / stock.square().mean().sqrt()) < 0.02
