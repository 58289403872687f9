"""Performance cases: the work that users of this package have it do, through its public entry points.

``listed()`` names one case per way the package is used; ``draw()`` samples the same ranges.  A case is
a dict of plain values whose ``"kind"`` says which entry point it exercises:

* ``linear``    one token through one bound ``PackedW3Linear``, called eagerly (HF ``generate`` style loops)
* ``linears``   the seven Linears of several decoder layers, one token, captured in one CUDA graph
* ``batch``     a few tokens (1..16) through ``w3_lut_gemv_out``, called eagerly
* ``hybrid``    one token through one bound ``PackedHybridLinear`` (two-base payload), called eagerly
* ``two_base``  the seven Linears of several layers in the row/column-scale two-base format, in one CUDA graph
* ``decode``    ``DecodeEngine``: a captured greedy continuation on an existing KV cache
* ``prefill``   ``DecodeEngine.prefill`` of a prompt
* ``fallback``  a prompt through ``PackedW3Linear`` with the dense fallback (prefill of the drop-in route)
* ``session``   ``StaticDecodeSession`` on a Hugging Face Qwen3 model with swapped Linears and fused modules
* ``convert``   a raw GPTQ W3 Linear on the host into the planar layout (checkpoint preparation)

Weights are synthetic with the value distributions of the decode benchmark: uniform codes, scales
U(0.005, 0.02), zero points 3 / 4, activations N(0, 1).  ``"checkpoint"`` selects what a GPTQ desc_act
checkpoint holds: bf16 scales, the constant zero point 4 and a column permutation; otherwise fp16
scales, stored zero points and identity order.
"""
import math

import torch

from marlin_style_fluxbin_b200.binary_global import global_two_base_m1_out
from marlin_style_fluxbin_b200.decode_engine import DecodeEngine, ModelShape
from marlin_style_fluxbin_b200.deployment import PackedHybridLinear
from marlin_style_fluxbin_b200.fused_modules import fused_qwen3_modules
from marlin_style_fluxbin_b200.gptq_deployment import convert_gptq_w3_to_planar
from marlin_style_fluxbin_b200.qwen3 import QWEN3_LINEAR_MODULES
from marlin_style_fluxbin_b200.static_decode import StaticDecodeSession, prepared_linears
from marlin_style_fluxbin_b200.w3_lut_deployment import PackedW3Linear, replace_w3_block_linears, w3_lut_gemv_out

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
SALIENT = 32  # dense residual columns of a two-base matrix

# Qwen3-8B widths.  Four of the 36 layers, and the vocabulary (151936 rows) cut in the same proportion,
# so that layers, attention and LM head keep their shares of a token while activations stay comparable
# between implementations: two 16-bit pipelines of this random-weight model part by 1.8 % in the logits
# after 4 layers, 2.8 % after 8 and 5 to 8 % after 36.
WIDTHS_8B = {"hidden": 4096, "q_heads": 32, "kv_heads": 8, "intermediate": 12288}
MODEL_8B = {"layers": 4, "vocab": 16896, **WIDTHS_8B}


def listed():
    return [
        # the smallest projection of a layer, token by token from Python: host latency and one short launch
        {"name": "linear_k_proj_eager", "kind": "linear", "out": 1024, "in": 4096, "dtype": "bf16", "checkpoint": True, "arithmetic": "structural"},
        # packed Linears under a captured decode step, module by module: the headline workload, weights larger than L2
        {"name": "linears_8b_graph", "kind": "linears", "layers": 8, "dtype": "bf16", "checkpoint": False, "arithmetic": "structural", **WIDTHS_8B},
        # four concurrent sequences (or a short draft) on a square projection
        {"name": "batch4_o_proj", "kind": "batch", "rows": 4, "out": 4096, "in": 4096, "dtype": "bf16", "checkpoint": False},
        # sixteen sequences on the widest projection: the largest small batch
        {"name": "batch16_gate_proj", "kind": "batch", "rows": 16, "out": 12288, "in": 4096, "dtype": "bf16", "checkpoint": False},
        # the two-base payload's module in a Python token loop
        {"name": "hybrid_q_proj_eager", "kind": "hybrid", "out": 4096, "in": 4096, "dtype": "bf16", "planar": True},
        # the two-base row/column-scale format under a captured step
        {"name": "two_base_8b_graph", "kind": "two_base", "layers": 4, "dtype": "bf16", **WIDTHS_8B},
        # the decode benchmark: 512 prompt tokens, 32 more in one graph
        {"name": "decode_512", "kind": "decode", "start": 512, "steps": 32, "dtype": "bf16", "arithmetic": "structural", **MODEL_8B},
        # a long conversation, with the arithmetic that follows the dequantised weights
        {"name": "decode_4096", "kind": "decode", "start": 4096, "steps": 16, "dtype": "bf16", "arithmetic": "decoded_bf16", **MODEL_8B},
        # time to first token of that prompt
        {"name": "prefill_512", "kind": "prefill", "tokens": 512, "dtype": "bf16", **MODEL_8B},
        # a ragged prompt through one swapped Linear of the drop-in route
        {"name": "fallback_333_up_proj", "kind": "fallback", "tokens": 333, "out": 12288, "in": 4096, "dtype": "bf16", "checkpoint": True},
        # the drop-in route's token loop: an unmodified Hugging Face model, whole continuation in one graph
        {"name": "session_8b", "kind": "session", "prompt": 128, "steps": 8, "checkpoint": True, **MODEL_8B},
        # preparing a checkpoint, one Linear
        {"name": "convert_k_proj", "kind": "convert", "out": 1024, "in": 4096, "desc_act": True},
    ]


def _log(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _widths(rng):
    """Layer widths from a tiny test model to Qwen3-32B's (hidden 5120, 64 heads, 25600), odd group counts included."""
    kv_heads = rng.choice((1, 2, 4, 8))
    q_heads = kv_heads * rng.choice((1, 2, 4, 5, 8))
    return {"hidden": 128 * _log(rng, 2, 40), "q_heads": q_heads, "kv_heads": kv_heads, "intermediate": 128 * max(q_heads, _log(rng, 3, 128))}


def _weights(case):
    return sum(out * inp for _, out, inp in _seven(case))


def draw(rng):
    kind = rng.choice(("linear", "linears", "batch", "batch", "hybrid", "two_base", "decode", "decode", "prefill", "fallback", "session", "convert"))
    case = {"kind": kind}
    matrix = {"out": 32 * _log(rng, 1, 800), "in": 128 * _log(rng, 1, 200)}
    if matrix["out"] * matrix["in"] > 12288 * 8192:
        matrix["in"] = 128 * max(1, 12288 * 8192 // matrix["out"] // 128)
    dtype = {"dtype": rng.choice(("bf16", "bf16", "fp16"))}
    checkpoint = {"checkpoint": rng.random() < 0.5}
    arithmetic = {"arithmetic": rng.choice(("structural", "structural", "decoded_bf16"))}
    if kind == "linear":
        case.update(matrix, **dtype, **checkpoint, **arithmetic)
    elif kind == "linears":
        case.update(layers=rng.randint(1, 6), **dtype, **checkpoint, **arithmetic, **_widths(rng))
    elif kind == "batch":
        case.update(rows=rng.randint(1, 16), **matrix, **dtype, **checkpoint)
    elif kind == "hybrid":
        out = _log(rng, 17, 12288)  # any number of rows, odd ones included
        case.update(out=out, planar=rng.random() < 0.6, **dtype)
        case["in"] = 128 * _log(rng, 1, 96 if out < 6000 else 32)
    elif kind == "two_base":
        case.update(layers=rng.randint(1, 4), **dtype, **_widths(rng))
    elif kind == "decode":
        case.update(layers=rng.randint(1, 4), vocab=rng.randint(500, 16896), start=_log(rng, 1, 4096), steps=rng.randint(2, 16), **dtype, **arithmetic, **_widths(rng))
    elif kind == "prefill":
        case.update(layers=rng.randint(1, 4), vocab=rng.randint(500, 16896), tokens=_log(rng, 2, 512), **dtype, **_widths(rng))
    elif kind == "fallback":
        case.update(tokens=_log(rng, 2, 1024), **matrix, **dtype, **checkpoint)
    elif kind == "session":
        case.update(prompt=_log(rng, 2, 512), steps=rng.randint(2, 8), layers=rng.randint(1, 3), vocab=rng.randint(500, 16896), **checkpoint, **_widths(rng))
    else:
        case.update({"out": 32 * _log(rng, 1, 32), "in": 128 * _log(rng, 1, 32)}, desc_act=rng.random() < 0.7)
    if "layers" in case:  # at most as many weights as the listed models
        case["layers"] = max(1, min(case["layers"], MODEL_8B["layers"] * _weights(WIDTHS_8B) // _weights(case)))
    return case


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _w3_layout(out, inp, gen, checkpoint):
    groups = inp // 128
    layout = {
        "planes": torch.randint(0, 256, (groups, 3, out, 16), dtype=torch.uint8, device="cuda", generator=gen),
        "scales": (torch.rand(groups, out, device="cuda", generator=gen) * 0.015 + 0.005).to(torch.bfloat16 if checkpoint else torch.float16),
    }
    if checkpoint:
        layout["perm"] = torch.randperm(inp, device="cuda", generator=gen).to(torch.int16)
    else:
        layout["zeros"] = torch.randint(3, 5, (groups, out), dtype=torch.uint8, device="cuda", generator=gen)
        layout["perm"] = torch.arange(inp, dtype=torch.int16, device="cuda")
    return layout


def _seven(case):
    hidden, q, kv, inter = case["hidden"], 128 * case["q_heads"], 128 * case["kv_heads"], case["intermediate"]
    return (("hidden", q, hidden), ("hidden", kv, hidden), ("hidden", kv, hidden), ("heads", hidden, q),
            ("mlp", inter, hidden), ("mlp", inter, hidden), ("inter", hidden, inter))


def _activations(case, gen, dtype):
    sizes = {"hidden": case["hidden"], "heads": 128 * case["q_heads"], "mlp": case["hidden"], "inter": case["intermediate"]}
    return {role: torch.randn(1, size, device="cuda", generator=gen).to(dtype) for role, size in sizes.items()}


def _graph_of(body):
    """``body`` warmed up and captured on a side stream: what a decode loop does once, before its first token."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.inference_mode(), torch.cuda.stream(stream):
        body()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            outputs = body()
    torch.cuda.current_stream().wait_stream(stream)
    return graph, outputs


def _prepare_linear(case, gen):
    dtype = DTYPES[case["dtype"]]
    module = PackedW3Linear(_w3_layout(case["out"], case["in"], gen, case["checkpoint"]), row_tile=256, arithmetic=case["arithmetic"])
    module.bind_prepared_decode(dtype)
    return {"module": module, "x": torch.randn(1, 1, case["in"], device="cuda", generator=gen).to(dtype)}


def _prepare_linears(case, gen):
    dtype = DTYPES[case["dtype"]]
    calls, keep = [], []
    for _ in range(case["layers"]):
        x = _activations(case, gen, dtype)
        for role, out, inp in _seven(case):
            module = PackedW3Linear(_w3_layout(out, inp, gen, case["checkpoint"]), row_tile=256, arithmetic=case["arithmetic"])
            module.bind_prepared_decode(dtype)
            calls.append((module, x[role].view(1, 1, -1)))
            keep.append(module)
    graph, outputs = _graph_of(lambda: [module(x) for module, x in calls])
    return {"graph": graph, "outputs": outputs, "keep": (calls, keep)}


def _prepare_batch(case, gen):
    dtype = DTYPES[case["dtype"]]
    return {"layout": _w3_layout(case["out"], case["in"], gen, case["checkpoint"]),
            "x": torch.randn(case["rows"], case["in"], device="cuda", generator=gen).to(dtype),
            "out": torch.empty(case["rows"], case["out"], device="cuda", dtype=dtype)}


def _prepare_hybrid(case, gen):
    out, groups, dtype = case["out"], case["in"] // 128, DTYPES[case["dtype"]]
    normal = lambda *size: torch.randn(*size, device="cuda", generator=gen)  # noqa: E731
    code = lambda *size: torch.randint(0, 256, size, dtype=torch.uint8, device="cuda", generator=gen)  # noqa: E731
    payload = {
        "global_sign_codes": code(out, groups * 32),
        "global_row_scales": normal(2, out, groups) * 0.1,
        "global_column_scales": normal(2, groups, 128),
        "refinement_indices": torch.rand(groups, 128, device="cuda", generator=gen).argsort(1)[:, :8].sort(1).values.to(torch.int16),
        "refinement_sign_codes": code(out, groups * 2),
        "refinement_row_scales": normal(2, out, groups) * 0.07,
        "refinement_column_scales": normal(2, groups, 8),
    }
    module = PackedHybridLinear(payload, kernel="v5_p1024" if case["planar"] else "v5", groups_per_split=1)
    module.bind_prepared_decode(dtype)
    return {"module": module, "x": normal(1, 1, case["in"]).to(dtype)}


def _prepare_two_base(case, gen):
    dtype = DTYPES[case["dtype"]]
    calls = []
    for _ in range(case["layers"]):
        x = _activations(case, gen, dtype)
        for role, out, inp in _seven(case):
            scale = lambda n: (torch.randn(2, n, device="cuda", generator=gen) * 0.02).abs().to(torch.float16)  # noqa: E731
            layout = {
                "codes": torch.randint(0, 256, (inp // 128, out, 2, 16), dtype=torch.uint8, device="cuda", generator=gen),
                "row_scales": scale(out),
                "column_scales": scale(inp),
                "salient_indices": torch.rand(inp, device="cuda", generator=gen).argsort()[:SALIENT].sort().values.to(torch.int32),
                "salient_values": (torch.randn(out, SALIENT, device="cuda", generator=gen) * 0.05).to(torch.bfloat16),
            }
            calls.append((x[role], layout, torch.empty(1, out, device="cuda", dtype=dtype)))
    graph, outputs = _graph_of(lambda: [global_two_base_m1_out(x, layout, out) for x, layout, out in calls])
    return {"graph": graph, "outputs": outputs, "keep": calls}


def _engine(case, seed, positions, **more):
    shape = ModelShape(case["layers"], case["hidden"], case["q_heads"], case["kv_heads"], 128, case["intermediate"], case["vocab"])
    return DecodeEngine(shape, device="cuda", max_positions=positions, seed=int(seed), dtype=DTYPES[case["dtype"]], **more)


def _prepare_decode(case, seed, gen):
    start, steps = case["start"], case["steps"]
    engine = _engine(case, seed, start + steps, arithmetic=case["arithmetic"])
    for cache in (engine.k_cache, engine.v_cache):  # the prompt's rows: k after its RMSNorm has unit scale
        cache[:, :, :start] = torch.randn(cache[:, :, :start].shape, device="cuda", generator=gen).to(cache.dtype)
    # the tokens are given (as in scoring a text), so that a near-tie between two logits cannot change what follows
    tokens = torch.randint(0, case["vocab"], (steps,), device="cuda", generator=gen)
    graph, _, logits = engine.capture(tokens[:1], start, steps, forced=tokens)
    return {"engine": engine, "graph": graph,
            "outputs": {"logits": logits, "keys": engine.k_cache[:, :, start:], "values": engine.v_cache[:, :, start:]}}


def _prepare_prefill(case, seed, gen):
    tokens = case["tokens"]
    engine = _engine(case, seed, tokens + 32)
    return {"engine": engine, "ids": torch.randint(0, case["vocab"], (1, tokens), device="cuda", generator=gen), "tokens": tokens}


def _prepare_fallback(case, gen):
    module = PackedW3Linear(_w3_layout(case["out"], case["in"], gen, case["checkpoint"]), row_tile=256, fallback="dense")
    return {"module": module, "x": torch.randn(1, case["tokens"], case["in"], device="cuda", generator=gen).to(DTYPES[case["dtype"]])}


def _prepare_session(case, seed, gen):
    from transformers import Qwen3Config, Qwen3ForCausalLM

    config = Qwen3Config(vocab_size=case["vocab"], hidden_size=case["hidden"], intermediate_size=case["intermediate"], num_hidden_layers=case["layers"],
                         num_attention_heads=case["q_heads"], num_key_value_heads=case["kv_heads"], head_dim=128, rope_theta=1e6, tie_word_embeddings=False)
    config._attn_implementation = "sdpa"
    default = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device("cuda"), torch.random.fork_rng(devices=[torch.cuda.current_device()]):
            torch.manual_seed(int(seed))
            model = Qwen3ForCausalLM(config).eval()
    finally:
        torch.set_default_dtype(default)
    for block in model.model.layers:
        payload, tiles = {}, {}
        for name in QWEN3_LINEAR_MODULES:
            old = block.get_submodule(name)
            layout = _w3_layout(old.out_features, old.in_features, gen, case["checkpoint"])
            payload.update({f"{name}.{field}": value for field, value in layout.items()})
            tiles[(old.out_features, old.in_features)] = 256
        replace_w3_block_linears(block, payload, fallback="dense", row_tile_by_shape=tiles)
    ids = torch.randint(0, case["vocab"], (1, case["prompt"]), device="cuda", generator=gen)
    forced = torch.randint(0, case["vocab"], (1, case["steps"]), device="cuda", generator=gen)
    with fused_qwen3_modules():
        session = StaticDecodeSession(model, ids, forced)
        binding = prepared_linears(model, torch.bfloat16)
        binding.__enter__()  # stays bound as long as the session lives
        session.capture()
    return {"session": session, "binding": binding}


def _prepare_convert(case, seed):
    gen = torch.Generator().manual_seed(int(seed))
    out, inp = case["out"], case["in"]
    word = lambda *size: torch.randint(-2**31, 2**31, size, dtype=torch.int64, generator=gen).to(torch.int32)  # noqa: E731
    order = torch.randperm(inp, generator=gen) if case["desc_act"] else torch.arange(inp)
    return {"qweight": word(3 * inp // 32, out), "qzeros": word(inp // 128, 3 * out // 32),
            "scales": (torch.rand(inp // 128, out, generator=gen) * 0.015 + 0.005).to(torch.float16), "g_idx": (order // 128).to(torch.int32)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "convert":
        return {"kind": kind, "tensors": _prepare_convert(case, seed)}
    gen = _generator(seed)
    maker = {"linear": _prepare_linear, "linears": _prepare_linears, "batch": _prepare_batch, "hybrid": _prepare_hybrid,
             "two_base": _prepare_two_base, "fallback": _prepare_fallback}.get(kind)
    state = maker(case, gen) if maker else {"decode": _prepare_decode, "prefill": _prepare_prefill, "session": _prepare_session}[kind](case, seed, gen)
    state["kind"] = kind
    return state


@torch.inference_mode()
def run(state):
    kind = state["kind"]
    if kind in ("linear", "hybrid", "fallback"):
        return state["module"](state["x"])
    if kind in ("linears", "two_base", "decode"):
        state["graph"].replay()
        return state["outputs"]
    if kind == "batch":
        return w3_lut_gemv_out(state["x"], state["layout"], state["out"])
    if kind == "prefill":
        engine, tokens = state["engine"], state["tokens"]
        logits = engine.prefill(state["ids"])
        return {"logits": logits, "keys": engine.k_cache[:, :, :tokens], "values": engine.v_cache[:, :, :tokens]}
    if kind == "session":
        session = state["session"]
        session.reset()
        session.graph.replay()
        return [logits for logits, _ in session.graph_outputs]
    return convert_gptq_w3_to_planar(state["tensors"], general=True)


def _w3_bytes(out, inp, checkpoint):
    groups = inp // 128
    return 3 * out * inp / 8 + 2 * groups * out + (2 * inp if checkpoint else groups * out)


def work(case):
    kind = case["kind"]
    if kind in ("linear", "batch", "fallback"):
        rows = {"linear": 1, "batch": case.get("rows"), "fallback": case.get("tokens")}[kind]
        out, inp = case["out"], case["in"]
        return {"bytes": _w3_bytes(out, inp, case["checkpoint"]) + 2 * rows * (out + inp), "flops": 2 * rows * out * inp}
    if kind == "hybrid":
        out, inp = case["out"], case["in"]
        groups = inp // 128
        # codes, fp32 row scales and refinement row scales, refinement codes, column scales, indices, activations
        return {"bytes": out * inp / 4 + groups * out * (8 + 8 + 2) + groups * (1024 + 64 + 16) + 2 * (out + inp), "flops": 4 * out * inp}
    if kind == "convert":
        out, inp = case["out"], case["in"]
        groups = inp // 128
        return {"bytes": 2 * (3 * out * inp / 8 + 2 * groups * out) + 3 * groups * out / 8 + groups * out + 4 * inp + 2 * inp, "flops": 0}
    matrices = [(out, inp) for _, out, inp in _seven(case)]
    weights = case["layers"] * _weights(case)
    if kind == "two_base":
        total = sum(out * inp / 4 + 4 * (out + inp) + 2 * SALIENT * out + 4 * SALIENT + 2 * (out + inp) for out, inp in matrices)
        return {"bytes": case["layers"] * total, "flops": 4 * weights}
    packed = case["layers"] * sum(_w3_bytes(out, inp, case.get("checkpoint", False)) for out, inp in matrices)
    if kind == "linears":
        return {"bytes": packed + case["layers"] * sum(2 * (out + inp) for out, inp in matrices), "flops": 2 * weights}
    head, cache_row = 2 * case["vocab"] * case["hidden"], 4 * case["layers"] * 128 * case["kv_heads"]  # k and v of one position, all layers
    score = 4 * 128 * case["q_heads"] * case["layers"]  # flops per (query, key) pair
    if kind == "prefill":
        tokens = case["tokens"]
        return {"bytes": packed + head + tokens * (cache_row + 2 * case["hidden"]),
                "flops": 2 * tokens * weights + score * tokens * tokens / 2 + head}
    start, steps = (case["start"], case["steps"]) if kind == "decode" else (case["prompt"], case["steps"])
    positions = steps * start + steps * (steps + 1) / 2
    total = {"bytes": steps * (packed + head + 4 * case["hidden"] + 2 * case["vocab"]) + positions * cache_row,
             "flops": steps * (2 * weights + head) + positions * score}
    if kind == "session":  # restoring the prompt's cache rows: read and written once
        total["bytes"] += 2 * start * cache_row
    return total


def tolerance(case):
    kind = case["kind"]
    if kind == "convert":
        return "exact"
    if kind in ("decode", "prefill", "session"):
        # a stack of layers in 16 bits: the roundings of two summation orders part after the first layer,
        # and the difference then grows with the depth as the distance of either from the exact result does
        return {"rel": 0.03}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
