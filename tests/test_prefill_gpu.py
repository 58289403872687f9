"""Many-token path: the dequantising kernel against the tensor-op restore of the same layout (bit for bit), its
row ranges and edges, and the packed Linear's dense fallback and the engine's prompts on every route: packed rows, the kernel that
dequantises into tensor memory, and one or several dense chunks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layout(o, k, *, scale_dtype, zeros, perm, seed):
    gen = torch.Generator().manual_seed(seed)
    groups = k // 128
    layout = {"planes": torch.randint(0, 256, (groups, 3, o, 16), generator=gen, dtype=torch.uint8),
              "scales": (torch.rand(groups, o, generator=gen) * 0.015 + 0.005).to(scale_dtype),
              "perm": (torch.randperm(k, generator=gen) if perm else torch.arange(k)).to(torch.int16)}
    if zeros:
        layout["zeros"] = torch.randint(0, 8, (groups, o), generator=gen, dtype=torch.uint8)
    return layout


@pytest.mark.parametrize("o,k,scale_dtype,zeros,perm", (
    (32, 128, torch.float16, False, False),      # half a 64-row block, one group
    (96, 640, torch.bfloat16, True, True),       # five groups: one beyond a walk of four
    (1024, 4096, torch.float16, True, False),
))
def test_dequantised_rows_equal_the_tensor_restore(o, k, scale_dtype, zeros, perm):
    from marlin_style_fluxbin_b200 import _native
    from marlin_style_fluxbin_b200.gptq_deployment import restore_planar_w3

    layout = _layout(o, k, scale_dtype=scale_dtype, zeros=zeros, perm=perm, seed=o + k)
    device = {name: value.cuda() for name, value in layout.items()}
    for dtype in (torch.bfloat16, torch.float16):
        want = restore_planar_w3(layout, dtype=dtype)  # host tensors: integer codes times scales
        assert torch.equal(restore_planar_w3(device, dtype=dtype).cpu(), want)
        part = torch.full((o - 32 + 1, k), float("nan"), device="cuda", dtype=dtype)[: o - 32] if o > 32 else None
        if part is not None:
            _native.w3_dequant([(device, part)], dtype, row_begin=16, row_count=o - 32)
            assert torch.equal(part.cpu(), want[16:o - 16][:, layout["perm"].long()])


@pytest.mark.parametrize("rows", (2, 4, 5, 16, 17, 100))
@pytest.mark.parametrize("perm,biased", ((False, False), (True, True), (True, False)))
def test_dense_fallback_of_the_packed_linear(rows, perm, biased):
    """Against x W^T + bias in fp32 of the restored weight: ONE rounding of the output to bf16's eight bits, at most half a
    unit in the last place = 2^-8 of the value, and fp32 sums of 1152 products (1152 x 2^-24 of the sum of magnitudes,
    below 2^-11 of the largest output here)."""
    from marlin_style_fluxbin_b200.gptq_deployment import restore_planar_w3
    from marlin_style_fluxbin_b200.w3_lut_deployment import PackedW3Linear

    layout = _layout(320, 1152, scale_dtype=torch.bfloat16, zeros=True, perm=perm, seed=rows)
    bias = torch.randn(320, generator=torch.Generator().manual_seed(3)).bfloat16() if biased else None
    x = torch.randn(1, rows, 1152, generator=torch.Generator().manual_seed(rows)).bfloat16()
    module = PackedW3Linear(layout, bias=bias, fallback="dense", row_tile=256).cuda()
    with torch.no_grad():
        got = module(x.cuda()).float().cpu()
    want = x.float() @ restore_planar_w3(layout, dtype=torch.float32).T
    if biased:
        want = want + bias.float()
    assert module.last_route == "dense_fallback" and got.shape == want.shape
    assert float((got - want).abs().max()) <= (2.0 ** -8 + 2.0 ** -11) * float(want.abs().max())


@pytest.mark.parametrize("tokens", (1, 3, 9, 17, 40))
def test_prefill_of_the_packed_arm_follows_the_dense_arm(tokens):
    """Both arms hold the same weights; logits and cache rows agree to 16-bit pipeline level (as the decode arms do)."""
    from marlin_style_fluxbin_b200.decode_engine import DecodeEngine, ModelShape

    shape = ModelShape(layers=2, hidden=384, q_heads=4, kv_heads=2, head_dim=128, intermediate=640, vocab=640)
    ids = torch.randint(0, 640, (1, tokens), generator=torch.Generator().manual_seed(tokens))
    found = {}
    for arm in ("bf16", "w3"):
        engine = DecodeEngine(shape, device="cuda", max_positions=48, arm=arm, seed=5)
        found[arm] = (engine.prefill(ids).float(), engine.k_cache[:, :, :tokens].float(), engine.v_cache[:, :, :tokens].float())
    for a, b in zip(found["w3"], found["bf16"]):
        assert bool(torch.isfinite(a).all()) and float((a - b).norm() / b.norm()) < 0.02


@pytest.mark.parametrize("rows", (16, 17, 333, 1024, 1025))
@pytest.mark.parametrize("perm,biased", ((False, False), (True, True)))
@pytest.mark.parametrize("chunk", (None, 1 << 20))
def test_dense_fallback_on_both_sides_of_its_routes(rows, perm, biased, chunk, monkeypatch):
    """2080 outputs: just wide enough for the kernel that dequantises into tensor memory, which ends at 1024 rows; 1 MB chunks leave
    five of them, the last one short.  Bound as in the test above, over 1152 products."""
    from marlin_style_fluxbin_b200 import w3_lut_deployment as w3
    from marlin_style_fluxbin_b200.gptq_deployment import restore_planar_w3

    assert w3.fused_gemm_pays(rows, 2080) == (rows <= 1024) and not w3.fused_gemm_pays(rows, 2048)
    if chunk is not None:
        monkeypatch.setattr(w3, "DENSE_CHUNK_BYTES", chunk)
        monkeypatch.setattr(w3, "fused_gemm_pays", lambda *_: False)
    layout = _layout(2080, 1152, scale_dtype=torch.bfloat16, zeros=True, perm=perm, seed=rows)
    bias = torch.randn(2080, generator=torch.Generator().manual_seed(3)).bfloat16() if biased else None
    x = torch.randn(1, rows, 1152, generator=torch.Generator().manual_seed(rows)).bfloat16()
    module = w3.PackedW3Linear(layout, bias=bias, fallback="dense", row_tile=256).cuda()
    with torch.no_grad():
        got = module(x.cuda()).float().cpu()
    want = x.float() @ restore_planar_w3(layout, dtype=torch.float32).T
    if biased:
        want = want + bias.float()
    assert float((got - want).abs().max()) <= (2.0 ** -8 + 2.0 ** -11) * float(want.abs().max())


@pytest.mark.parametrize("tokens,intermediate,chunk", (
    (40, 1152, None),        # gate and up through the kernel that dequantises into tensor memory
    (1040, 1152, None),      # beyond its rows: one dense chunk
    (40, 640, 200 << 10),    # several chunks, uneven ones: with the residual, and gate beside up
    (1040, 1152, 200 << 10),
))
def test_prefill_on_every_route_follows_the_dense_arm(tokens, intermediate, chunk, monkeypatch):
    from marlin_style_fluxbin_b200 import decode_engine, w3_lut_deployment

    if chunk is not None:
        monkeypatch.setattr(decode_engine, "DENSE_CHUNK_BYTES", chunk)
        monkeypatch.setattr(w3_lut_deployment, "DENSE_CHUNK_BYTES", chunk)
    shape = decode_engine.ModelShape(layers=2, hidden=384, q_heads=4, kv_heads=2, head_dim=128, intermediate=intermediate, vocab=640)
    ids = torch.randint(0, 640, (1, tokens), generator=torch.Generator().manual_seed(tokens))
    found = {}
    for arm in ("bf16", "w3"):
        engine = decode_engine.DecodeEngine(shape, device="cuda", max_positions=tokens + 8, arm=arm, seed=5)
        found[arm] = (engine.prefill(ids).float(), engine.k_cache[:, :, :tokens].float(), engine.v_cache[:, :, :tokens].float())
    for a, b in zip(found["w3"], found["bf16"]):
        assert bool(torch.isfinite(a).all()) and float((a - b).norm() / b.norm()) < 0.02
