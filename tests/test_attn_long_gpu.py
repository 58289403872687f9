"""Attention over long caches (two query heads a CTA) at the edges of its rounds, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_heads,kv_heads,length,dtype", (
    (4, 2, 640, torch.bfloat16),     # the last length of the first kernel
    (4, 2, 641, torch.bfloat16),     # the first of the long-cache kernel: chunks of 81 rows, the last of 74
    (4, 2, 647, torch.bfloat16),     # the last chunk one row short
    (32, 8, 1024, torch.bfloat16),   # whole rounds; 16 clusters do not fit at a time: merged through the scratch
    (10, 2, 1032, torch.float16),    # an odd group: a CTA with one head; one row in a second round
    (24, 8, 1032, torch.bfloat16),   # the same, merged through the scratch
    (10, 2, 1033, torch.float16),    # two rows in a second round, none in the last split's
    (5, 1, 3333, torch.bfloat16),    # a fourth round: the first stage is refilled
    (4, 2, 6145, torch.float16),     # a seventh of one row: all stages refilled, the first twice
    (32, 8, 8000, torch.bfloat16),
    (40, 8, 700, torch.bfloat16),    # 24 clusters, in two rounds
    (64, 8, 777, torch.float16),
    (8, 8, 1000, torch.bfloat16),    # nothing to share: the first kernel
    (30, 10, 2047, torch.bfloat16),  # more rounds of CTAs than the first kernel's: that one
    (30, 10, 2048, torch.bfloat16),
))
def test_long_cache(q_heads, kv_heads, length, dtype):
    from marlin_style_fluxbin_b200 import _native as nat
    from marlin_style_fluxbin_b200.decode_engine import synthetic_w3

    gen = torch.Generator(device="cuda").manual_seed(q_heads + length)
    normal = lambda *size: torch.randn(*size, device="cuda", generator=gen).to(dtype)  # noqa: E731
    q, k, v = normal(1, q_heads * 128), normal(1, kv_heads * 128), normal(1, kv_heads * 128)
    caches = [normal(kv_heads, length + 3, 128) for _ in range(2)]
    weights = [(1 + 0.1 * normal(128).float()).to(dtype) for _ in range(2)]
    angle = torch.rand(64, device="cuda", generator=gen).repeat(2) * 6
    cos, sin, scale = angle.cos().to(dtype), angle.sin().to(dtype), 128 ** -0.5
    scratch = torch.zeros(nat.attn_scratch_bytes(q_heads), dtype=torch.uint8, device="cuda")
    rotated = torch.empty(q_heads, 128, device="cuda", dtype=dtype)
    filled = [cache.clone() for cache in caches]
    nat.qknorm_rope_cache(q, k, v, *weights, cos, sin, rotated, *filled, length - 1, 1e-6)
    two = torch.empty(1, q_heads * 128, device="cuda", dtype=dtype)
    nat.attn_decode(rotated, *filled, two, length, scale, scratch)
    keys, values = (cache[:, :length].double() for cache in filled)
    scores = rotated.double().view(kv_heads, -1, 128) @ keys.transpose(1, 2) * scale
    share = scores.softmax(-1)
    want = share @ values
    # fp32: scores good to 128 x 2^-24 of their magnitudes, exponentials to as much again and 2^-21, sums of `length` terms; one rounding
    slack = 2.0 ** -24 * (2 * 128 * float((rotated.double().abs().view(kv_heads, -1, 128) @ keys.abs().transpose(1, 2)).max()) * scale + length + 8)
    bound = slack * (share @ values.abs()) + 2.0 ** (-8 if dtype == torch.bfloat16 else -11) * want.abs() + 2.0 ** -24
    assert bool(((two.double().view_as(want) - want).abs() <= bound).all())
    one = torch.empty_like(two)
    again = [cache.clone() for cache in caches]
    nat.attn_decode_fused(q, k, v, *weights, cos, sin, *again, one, length - 1, 1e-6, scale, scratch)
    assert torch.equal(one, two) and all(torch.equal(a, b) for a, b in zip(again, filled))
    # the pieces left for the o projection, merged here
    again = [cache.clone() for cache in caches]
    splits = nat.attn_decode_partial(q, k, v, *weights, cos, sin, *again, length - 1, 1e-6, scale, scratch)
    pieces = scratch[: q_heads * 16 * 132 * 4].view(torch.float32).view(q_heads, 16, 132)[:, :splits].double()
    factor = (pieces[..., 128] - pieces[..., 128].amax(1, keepdim=True)).exp()
    merged = (pieces[..., :128] * factor[..., None]).sum(1) / (pieces[..., 129] * factor).sum(1, keepdim=True)
    assert bool(((merged.view_as(want) - want).abs() <= bound).all()) and all(torch.equal(a, b) for a, b in zip(again, filled))
    # and by the o projection, which gets the bits of the whole launch
    layout = synthetic_w3(32, q_heads * 128, torch.device("cuda"), gen)
    results = []
    for merge in (True, False):
        y = torch.empty(1, 32, device="cuda", dtype=dtype)
        matrices = nat.w3_matrix_list([(layout["planes"], layout["scales"], layout["zeros"], y, None)])
        if merge:
            nat.w3_gemv_attn_merge(scratch, splits, dtype, q_heads * 128, matrices, 1, 32, torch.float16)
        else:
            nat.w3_gemv_multi(one, matrices, 1, 32, torch.float16, None)
        results.append(y)
    assert torch.equal(*results)


@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
def test_batches_are_summed_before_they_meet_the_sums(dtype):
    """Equal scores; a split's 256 positions hold one `large` value, and 2^-24 of it in the four positions that the same lane takes in its
    next batch.  One by one these are half a unit of the last place of `large` and lost to the rounding; together they are kept, and
    nothing else of the sums rounds."""
    from marlin_style_fluxbin_b200 import _native as nat

    q_heads, kv_heads, length = 4, 2, 2048
    large = 2.0 ** 14
    values = torch.zeros(8, 256, device="cuda", dtype=torch.float64)
    values[:, 0], values[:, 128::32] = large, large * 2.0 ** -24
    v_cache = values.reshape(1, length, 1).expand(kv_heads, length, 128).to(dtype).contiguous()
    assert torch.equal(v_cache[0, :, 0].double(), values.reshape(-1))  # 16 bits hold them
    k_cache = torch.zeros_like(v_cache)
    zeros = lambda n: torch.zeros(1, n, device="cuda", dtype=dtype)  # noqa: E731
    ones = torch.ones(128, device="cuda", dtype=dtype)
    scratch = torch.zeros(nat.attn_scratch_bytes(q_heads), dtype=torch.uint8, device="cuda")
    splits = nat.attn_decode_partial(zeros(q_heads * 128), zeros(kv_heads * 128), v_cache[:, -1].reshape(1, -1).contiguous(), ones, ones, ones, ones,
                                     k_cache, v_cache, length - 1, 1e-6, 128 ** -0.5, scratch)
    pieces = scratch[: q_heads * 16 * 132 * 4].view(torch.float32).view(q_heads, 16, 132)[:, :splits]
    assert splits == 8 and bool((pieces[..., 129] == 256).all())
    assert bool((pieces[..., :128].double() == large * (1 + 2.0 ** -22)).all())


@pytest.mark.parametrize("q_heads,kv_heads,length", ((4, 2, 1500), (32, 8, 700)))
def test_rows_off_a_16_byte_boundary(q_heads, kv_heads, length):
    """Caches on an 8-byte boundary are taken at any length (by the first kernel)."""
    from marlin_style_fluxbin_b200 import _native as nat

    gen = torch.Generator(device="cuda").manual_seed(length)
    normal = lambda *size: torch.randn(*size, device="cuda", generator=gen).bfloat16()  # noqa: E731
    q, caches = normal(1, q_heads * 128), []
    for _ in range(2):
        caches.append(normal(kv_heads * length * 128 + 4)[4:].view(kv_heads, length, 128))
        assert caches[-1].data_ptr() % 16 == 8
    scratch = torch.zeros(nat.attn_scratch_bytes(q_heads), dtype=torch.uint8, device="cuda")
    out = torch.empty_like(q)
    nat.attn_decode(q, *caches, out, length, 128 ** -0.5, scratch)
    share = (q.double().view(kv_heads, -1, 128) @ caches[0].double().transpose(1, 2) * 128 ** -0.5).softmax(-1)
    want = share @ caches[1].double()
    # the rounding of the result, and the fp32 sums far below it
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -14 * (share @ caches[1].double().abs())
    assert bool(((out.double().view_as(want) - want).abs() <= bound).all())


@pytest.mark.parametrize("q_heads,kv_heads,length,uses", (
    (28, 2, 700, False), (32, 8, 700, True), (32, 4, 5000, True), (36, 4, 5000, False), (40, 8, 700, False), (64, 8, 700, True), (64, 8, 600, False)))
def test_scratch_merges_only_where_clusters_need_more_rounds(q_heads, kv_heads, length, uses):
    """15 clusters of eight CTAs run at a time, 148 CTAs by themselves: the scratch is touched where that takes fewer rounds."""
    from marlin_style_fluxbin_b200 import _native as nat

    gen = torch.Generator(device="cuda").manual_seed(length)
    normal = lambda *size: torch.randn(*size, device="cuda", generator=gen).bfloat16()  # noqa: E731
    scratch = torch.zeros(nat.attn_scratch_bytes(q_heads), dtype=torch.uint8, device="cuda")
    q = normal(1, q_heads * 128)
    nat.attn_decode(q, normal(kv_heads, length, 128), normal(kv_heads, length, 128), torch.empty_like(q), length, 128 ** -0.5, scratch)
    assert bool(scratch.any()) == uses
    assert not scratch[q_heads * 16 * 132 * 4:].any()  # tickets are left zero
