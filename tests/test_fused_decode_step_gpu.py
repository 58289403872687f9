"""A session's decode steps with the one-launch attention and gate, against the same session on the stock modules."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,prompt", ((4, 2, 3), (5, 1, 80), (4, 4, 161)))
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
def test_fused_steps_follow_the_stock_modules(heads, kv_heads, prompt, dtype):
    """Prompt lengths around the 80 positions of one split; NRMSE of the logits at the level of a 16-bit pipeline (two
    layers, 2^-8 per rounding for bf16)."""
    from transformers import Qwen3Config, Qwen3ForCausalLM

    from marlin_style_fluxbin_b200.fused_modules import fused_qwen3_modules
    from marlin_style_fluxbin_b200.static_decode import StaticDecodeSession

    torch.manual_seed(heads)
    config = Qwen3Config(vocab_size=96, hidden_size=128, intermediate_size=256, num_hidden_layers=2, num_attention_heads=heads,
                         num_key_value_heads=kv_heads, head_dim=128)
    config._attn_implementation = "sdpa"
    model = Qwen3ForCausalLM(config).eval().cuda().to(dtype)
    ids = torch.randint(0, 96, (1, prompt), device="cuda")
    forced = torch.randint(0, 96, (1, 4), device="cuda")
    session = StaticDecodeSession(model, ids, forced)
    stock = session.audit()["logits"]
    rows = [layer.keys.clone() for layer in session.cache.layers]
    with fused_qwen3_modules():
        fused = session.audit()["logits"]
        for want, layer in zip(rows, session.cache.layers):  # the same cache rows, up to 16-bit roundings upstream
            assert float((layer.keys.float() - want.float()).norm() / want.float().norm()) < 0.02
        calls = []
        handle = model.model.layers[0].self_attn.q_norm.register_forward_hook(lambda *a: calls.append(1))
        session.audit()
        handle.remove()
        assert len(calls) == 4  # a hooked norm is called, not skipped
        graph = session.capture()["logits"]
        assert torch.equal(graph, fused) and torch.equal(session.measure("sequence_graph")[1]["logits"], fused)
    gap = (fused.float() - stock.float()).square().mean().sqrt() / stock.float().square().mean().sqrt()
    assert float(gap) < 0.02


@pytest.mark.parametrize("change", ("act_fn", "q_norm", "instance", "attention class"))
def test_replaced_parts_run_as_they_are(change):
    """A session on a model whose parts were exchanged: the fused steps equal the stock ones, with those parts in them."""
    from transformers import Qwen3Config, Qwen3ForCausalLM
    from transformers.models.qwen3 import modeling_qwen3

    from marlin_style_fluxbin_b200.fused_modules import fused_qwen3_modules
    from marlin_style_fluxbin_b200.static_decode import StaticDecodeSession

    torch.manual_seed(2)
    config = Qwen3Config(vocab_size=96, hidden_size=128, intermediate_size=256, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=128)
    config._attn_implementation = "sdpa"
    model = Qwen3ForCausalLM(config).eval().cuda().bfloat16()
    with torch.no_grad():
        for weight in model.parameters():  # so that the exchanged parts show in the logits
            weight.mul_(8 if weight.ndim == 2 else 1)
    for block in model.model.layers:
        attention, mlp = block.self_attn, block.mlp
        if change == "act_fn":
            mlp.act_fn = torch.nn.GELU()
        elif change == "q_norm":
            attention.q_norm = torch.nn.RMSNorm(128, eps=1.0).to(attention.k_norm.weight)
        elif change == "instance":
            attention.k_norm.forward = lambda x, norm=attention.k_norm: type(norm).forward(norm, x) * 3
        else:
            class Doubled(modeling_qwen3.Qwen3Attention):
                def forward(self, *args, **kwargs):
                    heads, weights = super().forward(*args, **kwargs)
                    return heads * 2, weights

            attention.__class__ = Doubled
    ids, forced = torch.randint(0, 96, (1, 5), device="cuda"), torch.randint(0, 96, (1, 3), device="cuda")
    session = StaticDecodeSession(model, ids, forced)
    stock = session.audit()["logits"].float()
    with fused_qwen3_modules():
        fused = session.audit()["logits"].float()
    assert float((fused - stock).square().mean().sqrt() / stock.square().mean().sqrt()) < 0.02


def test_hooks_on_every_module_see_every_module():
    from transformers import Qwen3Config, Qwen3ForCausalLM

    from marlin_style_fluxbin_b200.fused_modules import fused_qwen3_modules
    from marlin_style_fluxbin_b200.static_decode import StaticDecodeSession

    config = Qwen3Config(vocab_size=96, hidden_size=128, intermediate_size=256, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, head_dim=128)
    config._attn_implementation = "sdpa"
    model = Qwen3ForCausalLM(config).eval().cuda().bfloat16()
    session = StaticDecodeSession(model, torch.randint(0, 96, (1, 5), device="cuda"), torch.randint(0, 96, (1, 2), device="cuda"))
    seen = []
    handle = torch.nn.modules.module.register_module_forward_hook(lambda module, *a: seen.append(module))
    try:
        with fused_qwen3_modules():
            session.audit()
    finally:
        handle.remove()
    block = model.model.layers[0]
    assert all(sum(module is part for module in seen) == 2 for part in (block.self_attn.q_norm, block.self_attn.k_norm, block.mlp.act_fn, block.mlp))
