"""Single-kernel RMSNorm and rotary embedding for the stock HF Qwen3 decode path.

Mirror of the reference's ``fused_modules`` (``src/fluxbin_style/fused_modules.py:30-112``):
same function names and the same context manager that patches
``Qwen3RMSNorm.forward`` and ``modeling_qwen3.apply_rotary_pos_emb`` and restores them on exit.
The reference gets its RMSNorm fusion from ``torch.compile`` and its RoPE from tensor algebra;
here both are hand-written sm_100a kernels behind the C ABI (``fb_rmsnorm``, ``fb_rope_qk``).
The kernels serve CUDA fp16/bf16 tensors; the one-position RoPE kernel serves decode steps.
Anything else (CPU tensors, fp32, prefill with many positions) runs the same mathematics as
plain tensor operations, which is also what the patched functions compute in the reference.
"""
from __future__ import annotations

import inspect
import threading
from contextlib import contextmanager

import torch
from torch.nn.modules import module as module_base

from . import _native
from .w3_lut_deployment import PackedW3Linear


def rms_norm_reference(hidden_states, weight, eps):
    """The stock Qwen3RMSNorm arithmetic as a free function (fp32 statistics, cast, then weight)."""
    dtype = hidden_states.dtype
    wide = hidden_states.to(torch.float32)
    wide = wide * torch.rsqrt(wide.pow(2).mean(-1, keepdim=True) + eps)
    return weight * wide.to(dtype)


def _kernel_eligible(*tensors) -> bool:
    first = tensors[0]
    return (first.is_cuda and first.dtype in (torch.float16, torch.bfloat16) and not torch.is_grad_enabled()
            and all(t.is_cuda and t.dtype == first.dtype and t.is_contiguous() for t in tensors))


def fused_rms_norm(hidden_states, weight, eps):
    """RMSNorm in one kernel launch when the tensors are CUDA 16-bit, else the reference math."""
    if not _kernel_eligible(hidden_states, weight) or weight.numel() != hidden_states.shape[-1]:
        return rms_norm_reference(hidden_states, weight, eps)
    out = torch.empty_like(hidden_states)
    _native.rmsnorm(hidden_states, weight, out, eps)
    return out


def fused_rms_norm_forward(self, hidden_states):
    return fused_rms_norm(hidden_states, self.weight, self.variance_epsilon)


def _rope_algebra(q, k, cos, sin, unsqueeze_dim):
    cos, sin = cos.unsqueeze(unsqueeze_dim), sin.unsqueeze(unsqueeze_dim)
    q_heads = q.shape[unsqueeze_dim]
    both = torch.cat((q, k), dim=unsqueeze_dim)
    half = both.shape[-1] // 2
    turned = torch.cat((-both[..., half:], both[..., :half]), dim=-1)
    result = torch.addcmul(both * cos, turned, sin)
    return result.narrow(unsqueeze_dim, 0, q_heads), result.narrow(unsqueeze_dim, q_heads, k.shape[unsqueeze_dim])


def fused_apply_rotary_pos_emb(q, k, cos, sin, unsqueeze_dim=1):
    """Rotate q and k together.  One kernel for a single position on CUDA, tensor algebra otherwise."""
    if q.ndim != k.ndim or q.dtype != k.dtype or q.shape[-1] != k.shape[-1]:
        raise ValueError("fused RoPE requires q/k with matching rank, dtype and head_dim")
    dim = q.shape[-1]
    single_position = cos.numel() == dim and sin.numel() == dim and q.numel() == q.shape[unsqueeze_dim] * dim \
        and k.numel() == k.shape[unsqueeze_dim] * dim
    if single_position and dim % 2 == 0 and _kernel_eligible(q, k, cos, sin):
        q_out, k_out = torch.empty_like(q), torch.empty_like(k)
        _native.rope_qk(q, k, cos, sin, q_out, k_out)
        return q_out, k_out
    return _rope_algebra(q, k, cos, sin, unsqueeze_dim)


# ---- one decode step on a static cache (StaticDecodeSession) ----
# Between the Linears of a step lie some seventeen small launches per layer in the stock modules: norms and rotation,
# two scatters into the cache and their index arithmetic, the expansion of the k/v heads, SDPA, gate and product.  While a
# session announces the step it runs (position and cache known on the host), the attention module takes ONE launch
# for everything between q/k/v and o_proj, and the MLP one between gate/up and down.  Bound W3 projections o_proj and
# down_proj also add the residual in their launch: two of thirteen launches of a layer, 4 % of a step.
_local = threading.local()


def _qwen3():
    from transformers.models.qwen3 import modeling_qwen3

    return modeling_qwen3


def _activations():
    from transformers.activations import ACT2FN

    return ACT2FN


class DecodeStep:
    """What a session tells the modules about the step under way; ``position`` advances from step to step."""

    def __init__(self, cache, scratch):
        self.cache, self.scratch, self.position = cache, scratch, None

    @contextmanager
    def at(self, position: int):
        self.position, previous, _local.step = position, getattr(_local, "step", None), self
        try:
            yield
        finally:
            _local.step = previous


def _runs(module, *classes) -> bool:
    """Whether calling ``module`` runs the forward of one of these classes and nothing else, so that a fused launch may stand
    for it: no class or instance of its own making, no hooks on it or on every module, no compiled call."""
    return (any(getattr(type(module), "forward", None) is owner.forward for owner in classes) and "forward" not in module.__dict__
            and getattr(module, "_compiled_call_impl", None) is None
            and not (module._forward_hooks or module._forward_pre_hooks or module_base._global_forward_hooks or module_base._global_forward_pre_hooks))


def _step_serves(step, attention, call) -> bool:
    hidden, positions = call.get("hidden_states"), call.get("position_embeddings")
    if call.get("past_key_values", call.get("past_key_value")) is not step.cache or positions is None:
        return False
    q_norm, k_norm = attention.q_norm, attention.k_norm
    if not _runs(q_norm, _qwen3().Qwen3RMSNorm) or not _runs(k_norm, _qwen3().Qwen3RMSNorm):
        return False
    layer = step.cache.layers[attention.layer_idx]
    keys, values = layer.keys, layer.values
    dim = attention.head_dim
    return (dim == 128 and hidden.numel() == hidden.shape[-1] and attention.config._attn_implementation == "sdpa"
            and getattr(attention, "sliding_window", None) is None and not attention.training
            and not call.get("output_attentions") and not call.get("kwargs", {}).get("output_attentions")
            and positions[0].numel() == dim and _kernel_eligible(hidden, q_norm.weight, k_norm.weight, *positions, keys, values)
            and q_norm.variance_epsilon == k_norm.variance_epsilon and keys.shape == values.shape and keys.shape[0] == 1 and keys.shape[-1] == dim
            and step.position < keys.shape[2] and attention.config.num_attention_heads % keys.shape[1] == 0
            and step.scratch.numel() >= _native.attn_scratch_bytes(attention.config.num_attention_heads))


def _attention_heads(step, attention, call):
    """What o_proj takes, in one launch behind q/k/v; None where that launch does not serve."""
    if not _step_serves(step, attention, call):
        return None
    hidden, (cos, sin) = call["hidden_states"], call["position_embeddings"]
    q, k, v = attention.q_proj(hidden), attention.k_proj(hidden), attention.v_proj(hidden)
    if not _kernel_eligible(hidden, q, k, v):
        return None
    layer, out = step.cache.layers[attention.layer_idx], torch.empty_like(q)
    _native.attn_decode_fused(q, k, v, attention.q_norm.weight, attention.k_norm.weight, cos, sin, layer.keys[0], layer.values[0], out,
                              step.position, attention.q_norm.variance_epsilon, attention.scaling, step.scratch)
    return out


def _gates(mlp) -> bool:
    return _runs(mlp.act_fn, torch.nn.SiLU, type(_activations()["silu"]))


def _gated(mlp, x):
    """What down_proj takes, in one launch behind gate/up; None where that launch does not serve."""
    if not _gates(mlp) or not _kernel_eligible(x):
        return None
    gate, up = mlp.gate_proj(x), mlp.up_proj(x)
    if not _kernel_eligible(x, gate, up):
        return None
    out = torch.empty_like(gate)
    _native.silu_mul(gate, up, out)
    return out


def _fused_attention(original):
    signature = inspect.signature(original)

    def forward(self, *args, **kwargs):
        step = getattr(_local, "step", None)
        heads = None if step is None else _attention_heads(step, self, signature.bind(self, *args, **kwargs).arguments)
        return original(self, *args, **kwargs) if heads is None else (self.o_proj(heads), None)

    return forward


def _fused_mlp(original):
    def forward(self, x):
        act = None if getattr(_local, "step", None) is None else _gated(self, x)
        return original(self, x) if act is None else self.down_proj(act)

    return forward


def _joins(projection) -> bool:
    """Whether a projection can take the residual addition that follows it into its launch."""
    return _runs(projection, PackedW3Linear) and projection._decode_binding is not None and projection.bias is None


def _fused_layer(original):
    signature = inspect.signature(original)

    def forward(self, *args, **kwargs):
        step, attention, mlp = getattr(_local, "step", None), self.self_attn, self.mlp
        if step is None or not (_runs(attention, _qwen3().Qwen3Attention) and _runs(mlp, _qwen3().Qwen3MLP) and _joins(attention.o_proj) and _joins(mlp.down_proj)):
            return original(self, *args, **kwargs)
        call = dict(signature.bind(self, *args, **kwargs).arguments)
        residual = call["hidden_states"]
        # both halves have to serve before anything is launched
        if not _step_serves(step, attention, call) or not _gates(mlp) or not _kernel_eligible(residual):
            return original(self, *args, **kwargs)
        call["hidden_states"] = self.input_layernorm(residual)
        heads = _attention_heads(step, attention, call)
        if heads is None or not attention.o_proj.adds_residual(heads):
            return original(self, *args, **kwargs)
        middle = attention.o_proj.add_to(residual, heads)
        normed = self.post_attention_layernorm(middle)
        act = _gated(mlp, normed)
        if act is None or not mlp.down_proj.adds_residual(act):
            return middle + mlp(normed)
        return mlp.down_proj.add_to(middle, act)

    return forward


@contextmanager
def fused_qwen3_modules(*, rms_norm=True, rope=True):
    """Patch the HF Qwen3 RMSNorm class and rotary function in place; restore on exit or error.

    The patch is at class / module scope on purpose, so every arm of a comparison built
    from ``transformers`` shares the same non-Linear path.  With both parts on, the decode steps of a
    ``StaticDecodeSession`` also take the attention and the SwiGLU gate in one launch each.
    """
    from transformers.models.qwen3 import modeling_qwen3

    applied = {"rms_norm": bool(rms_norm), "rope": bool(rope)}
    saved = {}
    try:
        if rms_norm:
            saved["rms_norm"] = modeling_qwen3.Qwen3RMSNorm.forward
            modeling_qwen3.Qwen3RMSNorm.forward = fused_rms_norm_forward
        if rope:
            saved["rope"] = modeling_qwen3.apply_rotary_pos_emb
            modeling_qwen3.apply_rotary_pos_emb = fused_apply_rotary_pos_emb
        if rms_norm and rope:
            for name, wrap in (("Qwen3Attention", _fused_attention), ("Qwen3MLP", _fused_mlp), ("Qwen3DecoderLayer", _fused_layer)):
                owner = getattr(modeling_qwen3, name)
                # layers of some transformers versions return a tuple; the fused one returns the hidden states alone
                if wrap is _fused_layer and inspect.signature(owner.forward).return_annotation not in (torch.Tensor, "torch.Tensor"):
                    continue
                saved[name] = owner.forward
                owner.forward = wrap(owner.forward)
        yield applied
    finally:
        if "rms_norm" in saved:
            modeling_qwen3.Qwen3RMSNorm.forward = saved["rms_norm"]
        if "rope" in saved:
            modeling_qwen3.apply_rotary_pos_emb = saved["rope"]
        for name in ("Qwen3Attention", "Qwen3MLP", "Qwen3DecoderLayer"):
            if name in saved:
                getattr(modeling_qwen3, name).forward = saved[name]
