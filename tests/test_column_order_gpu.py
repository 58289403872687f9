"""Whether a column order is the identity is asked on the stream and answered later: no answer may serve another question."""
import time
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replaced", (False, True))
def test_a_late_answer_is_not_taken_for_the_next_question(replaced):
    """The order is asked about, then changes (in place, or by another tensor that gets the address) and is asked about again, all
    queued behind one delay; behind a second one the first answer is there and the second is not."""
    from marlin_style_fluxbin_b200 import _native, w3_lut_deployment as w3

    gen = torch.Generator(device="cuda").manual_seed(3)
    o, k = 96, 640
    layout = {"planes": torch.randint(0, 256, (k // 128, 3, o, 16), dtype=torch.uint8, device="cuda", generator=gen),
              "scales": (torch.rand(k // 128, o, device="cuda", generator=gen) * 0.015 + 0.005).half(),
              "perm": torch.arange(k, dtype=torch.int16, device="cuda")}
    shuffled = torch.randperm(k, device="cuda", generator=gen).to(torch.int16)
    x = torch.randn(1, k, device="cuda", generator=gen).bfloat16()
    want, first, second, third = (torch.empty(1, o, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    _native.w3_gemv(x, layout["planes"], layout["scales"], None, shuffled, want)
    w3._perm_or_none(shuffled)  # the first question allocates
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # some 50 ms
    w3._perm_or_none(layout["perm"], wait=False)
    if replaced:
        del layout["perm"]
        layout["perm"] = shuffled.clone()
    else:
        layout["perm"].copy_(shuffled)
    torch.cuda._sleep(1_000_000_000)
    assert w3._perm_or_none(layout["perm"], wait=False) is layout["perm"]
    time.sleep(0.2)
    for out in (first, second, third):  # plain, prepared there and then, prepared
        w3.w3_lut_gemv_out(x, layout, out)
    assert all(torch.equal(out, want) for out in (first, second, third))


def test_questions_of_many_threads_through_full_blocks(monkeypatch):
    from marlin_style_fluxbin_b200 import w3_lut_deployment as w3

    monkeypatch.setattr(w3, "_MAX_PERMS", 8)
    monkeypatch.setattr(w3, "_perm_blocks", [])
    monkeypatch.setattr(w3, "_perm_given", 0)
    monkeypatch.setattr(w3, "_IDENTITY_PERMS", {})
    orders = [torch.arange(256, dtype=torch.int16, device="cuda") for _ in range(48)]
    for order in orders[::2]:
        order[:2] = order[:2].flip(0)
    torch.cuda.synchronize()
    with ThreadPoolExecutor(8) as pool:
        found = list(pool.map(lambda order: w3._perm_or_none(order) is None, orders))
    assert found == [index % 2 == 1 for index in range(48)]
    assert len(w3._perm_blocks) < 6  # full blocks went once their answers were there
