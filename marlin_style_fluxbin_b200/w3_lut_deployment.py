"""W3 GEMV operator wrappers and the ``nn.Linear`` replacement for batch-1 decode.

Mirror of the reference's ``w3_lut_deployment`` module (reference file
``src/fluxbin_style/w3_lut_deployment.py``): same public names, argument meaning and
error behaviour, so code written against the reference runs unchanged.  What differs is
underneath: one ahead-of-time built sm_100a library reached through a C ABI instead of
per-row-tile JIT extensions.  ``row_tile``, ``groups_per_split`` and the ``workspace``
argument are still validated exactly as before but are advisory: the kernel chooses its
own tiling, reduces its K split internally and leaves a caller's workspace untouched
(the two-call form ``inline_main`` + ``finish`` does fill it, one row per group).
"""
from __future__ import annotations

import threading
import weakref
from types import SimpleNamespace

import torch
from torch import nn
from torch.nn import functional as F

from . import _native
from .gptq_deployment import FIELDS, OPTIONAL_FIELDS, restore_planar_w3, validate_planar_w3

# A dense weight is formed and multiplied in row chunks of at most this size: the GEMM then reads the
# chunk out of the L2 (126 MB), and the next chunk overwrites it there before it is written back.
DENSE_CHUNK_BYTES = 52 << 20


def fused_gemm_pays(rows: int, out_features: int) -> bool:
    """Whether ``rows`` activation rows go through the kernel that dequantises into tensor memory rather than through dense
    chunks.  One tile of it walks all of K, so a narrow matrix keeps few SMs busy.  us in a graph, weights cold, bf16 activations, fp16 scales, this / chunks,
    512 rows: 512 x 4096 15.5 / 11.5, 1024 x 4096 15.6 / 12.9, 2048 x 4096 16.7 / 16.9, 2048 x 12288 40.0 / 35.7, 3072 x 4096 17.8 / 19.2, 3072 x 12288
    41.7 / 55.9, 4096 x 4096 18.7 / 22.4, 12288 x 4096 42.3 / 61.9; 64 rows: 2048 x 4096 15.4 / 14.1, 3072 x 4096 15.6 / 15.3, 4096 x 4096 15.7 / 16.3,
    12288 x 4096 16.4 / 38.8 (bf16 scales: 0.5 to 1.5 less for this below 256 rows).  Beyond a thousand rows the chunks, dequantised once for all of them, catch up where K is short: 2048
    rows of 12288 x 1024 49.5 / 48.4, but of 12288 x 4096 154 / 166.  Nor does the line follow K on its other side: 512 rows of 1024 x 1024 take 6.9 / 8.1."""
    return rows <= 1024 and out_features > 2048 and out_features % 32 == 0

ROW_TILES = (256, 512, 1024)
EXPERIMENTAL_ROW_TILES = ROW_TILES + (2048,)
ARITHMETIC_MODES = ("structural", "decoded_bf16")
QWEN3_ROW_TILE_BY_SHAPE = {
    (4096, 4096): 256,
    (1024, 4096): 512,
    (12288, 4096): 1024,
    (4096, 12288): 1024,
}
_OBSERVED_EXACT_SPLIT = {(4096, 4096): 1, (1024, 4096): 1, (12288, 4096): 4, (4096, 12288): 2}


def _route_table(arithmetic: str, split_of=lambda shape: 1) -> dict:
    return {
        shape: {"row_tile": tile, "groups_per_split": split_of(shape), "arithmetic": arithmetic}
        for shape, tile in QWEN3_ROW_TILE_BY_SHAPE.items()
    }


QWEN3_W3_ROUTE_POLICIES = {
    "structural": _route_table("structural"),
    "fast_corrected": _route_table("decoded_bf16"),
    "observed_exact": _route_table("decoded_bf16", _OBSERVED_EXACT_SPLIT.__getitem__),
}


def w3_lut_extension_build(row_tile: int, uniform_index_probe: bool = False):
    """Describe the native build that serves ``row_tile``.

    The reference compiles one extension per row tile; here every row tile maps to the
    same prebuilt library, so the "build" is a description: ``(kwargs, contract)``.
    A timing-only wrong-result probe build does not exist in this library.
    """
    if row_tile not in EXPERIMENTAL_ROW_TILES:
        raise ValueError(f"row_tile must be one of {EXPERIMENTAL_ROW_TILES}")
    if uniform_index_probe:
        raise ValueError("the uniform-index timing probe is not part of this library")
    from .build import ARCH, COMMON, CSRC, EXTRA, LIBRARY

    kwargs = {
        "name": "fluxbin_b200",
        "sources": [str(CSRC / "fb_w3_gemv.cu")],
        "extra_cuda_cflags": [*ARCH, *COMMON, *EXTRA["fb_w3_gemv.cu"]],
    }
    contract = {"library": str(LIBRARY), "row_tile": row_tile, "row_tile_is_advisory": True}
    return kwargs, contract


def load_w3_lut_extension(row_tile: int, uniform_index_probe: bool = False):
    """Return an object with the reference extension's four entry points.

    ``inline_main``, ``inline_main_bf16_weight``, ``finish`` and ``m1_out`` take the same
    positional tensors as the reference's pybind functions (csrc/w3_lut.cu:334-339).
    """
    if row_tile not in EXPERIMENTAL_ROW_TILES:
        raise ValueError(f"row_tile must be one of {EXPERIMENTAL_ROW_TILES}")
    if uniform_index_probe:
        raise ValueError("the uniform-index timing probe is not part of this library")
    if not torch.cuda.is_available():
        raise RuntimeError("W3 LUT requires NVIDIA CUDA; no CPU/MPS substitution")
    _native.library()

    def _partials(x, planes, scales, perm, partial, corrected):
        _check_native_args(x, planes, scales, perm, partial, planes.shape[0])
        _native.w3_gemv(x, planes, scales, None, _perm_or_none(perm), partial,
                        decoded_bf16=corrected, group_partials=True)

    def inline_main(x, planes, scales, perm, partial):
        _partials(x, planes, scales, perm, partial, False)

    def inline_main_bf16_weight(x, planes, scales, perm, partial):
        _partials(x, planes, scales, perm, partial, True)

    def finish(partial, out):
        if partial.ndim != 2 or partial.dtype != torch.float32 or not partial.is_cuda:
            raise RuntimeError("partial must be CUDA FP32 [G,O]")
        if tuple(out.shape) != (1, partial.shape[1]) or out.dtype not in (torch.float16, torch.bfloat16):
            raise RuntimeError("out must be FP16/BF16 [1,O]")
        _native.w3_finish(partial, out)

    def m1_out(x, planes, scales, perm, partial, out, groups_per_split, dense_bf16_weight_semantics):
        groups = planes.shape[0]
        if not 0 < groups_per_split <= 255:
            raise RuntimeError("groups_per_split outside v1 bounds")
        _check_native_args(x, planes, scales, perm, partial, -(-groups // groups_per_split))
        if tuple(out.shape) != (1, planes.shape[2]) or out.dtype != x.dtype or out.device != x.device:
            raise RuntimeError("out must be contiguous same-device [1,O] with input dtype")
        _native.w3_gemv(x, planes, scales, None, _perm_or_none(perm), out,
                        decoded_bf16=bool(dense_bf16_weight_semantics))

    return SimpleNamespace(inline_main=inline_main, inline_main_bf16_weight=inline_main_bf16_weight,
                           finish=finish, m1_out=m1_out)


# Whether a perm tensor is the identity (the kernels then skip the gather).  A kernel compares it on the stream and
# writes the answer to a word of pinned host memory, so that asking costs no wait: -1 until it has run.  Keyed by address,
# and an entry holds only while the tensor it was made for lives unchanged (another one may get the address later).
# Every question has a word of its own: an older one, about a tensor that was there before or about values since
# overwritten, may still be queued on some stream of some device, and its answer must not pass for the newer one's.
_IDENTITY_PERMS: dict[tuple[int, int], tuple] = {}
_MAX_PERMS = 4096
_perm_lock = threading.Lock()
_perm_blocks: list = []  # blocks of words: the last gives them out, those before it are full and still wait for answers
_perm_given = 0          # words of the last block


def _perm_entry(perm: torch.Tensor):
    """``(owner, version, words, index)`` of a perm that was asked about, or None."""
    entry = _IDENTITY_PERMS.get((perm.data_ptr(), perm.numel()))
    if entry is None or entry[0]() is not (perm if perm._base is None else perm._base) or entry[1] != (None if perm.is_inference() else perm._version):
        return None
    return entry


def _answer_word():
    """A word that no question has had, under the lock: ``(words, index, address)``."""
    global _perm_given
    if not _perm_blocks or _perm_given == _MAX_PERMS:
        # a full block whose answers are all there can go; entries keep the one they read
        _perm_blocks[:] = [block for block in _perm_blocks if int(block[0].min()) < 0]
        words = torch.full((_MAX_PERMS,), -1, dtype=torch.int32, pin_memory=torch.cuda.is_available())
        _perm_blocks.append((words.numpy(), words.data_ptr()))
        _perm_given = 0
        for key in [key for key, entry in _IDENTITY_PERMS.items() if entry[0]() is None]:
            del _IDENTITY_PERMS[key]
        if len(_IDENTITY_PERMS) >= _MAX_PERMS:
            _IDENTITY_PERMS.clear()
    words, address = _perm_blocks[-1]
    _perm_given += 1
    return words, _perm_given - 1, address + 4 * (_perm_given - 1)


def _ask_perm(perm: torch.Tensor):
    with _perm_lock:
        entry = _perm_entry(perm)  # another thread may have asked meanwhile
        if entry is not None:
            return entry
        words, index, address = _answer_word()
        try:
            with torch.cuda.device(perm.device):
                _native.check(_native.library().fb_identity_order(perm.data_ptr(), perm.numel(), address, _native.stream_handle(perm.device)))
        except BaseException:
            words[index] = 0  # nothing will answer
            raise
        entry = (weakref.ref(perm if perm._base is None else perm._base), None if perm.is_inference() else perm._version, words, index)
        _IDENTITY_PERMS[(perm.data_ptr(), perm.numel())] = entry
        return entry


def _perm_or_none(perm: torch.Tensor, wait: bool = True):
    """``None`` when ``perm`` is the identity.  ``perm`` itself, which is always valid, when it is not, or when that is not
    known yet and must not (a capture) or need not (``wait``) be waited for."""
    entry = _perm_entry(perm)
    if entry is None:
        if torch.cuda.is_current_stream_capturing():
            return perm
        entry = _ask_perm(perm)
    words, index = entry[2:]
    known = int(words[index])
    if known < 0 and wait and not torch.cuda.is_current_stream_capturing():
        torch.cuda.current_stream(perm.device).synchronize()
        known = int(words[index])
    return None if known == 1 else perm


def _check_native_args(x, planes, scales, perm, partial, splits) -> None:
    """The reference extension's argument contract (csrc/w3_lut.cu:191-226), as RuntimeError."""
    if not (x.is_cuda and x.is_contiguous() and x.ndim == 2 and x.shape[0] == 1):
        raise RuntimeError("CUDA x [1,K] required")
    for tensor in (planes, scales, perm, partial):
        if not (tensor.is_cuda and tensor.device == x.device and tensor.is_contiguous()):
            raise RuntimeError("all tensors must be contiguous on the input CUDA device")
    if x.dtype not in (torch.float16, torch.bfloat16):
        raise RuntimeError("x must be FP16 or BF16")
    if planes.dtype != torch.uint8 or planes.ndim != 4 or planes.shape[1] != 3 or planes.shape[3] != 16:
        raise RuntimeError("planes must be uint8 [G,3,O,16]")
    groups, _, out_features, _ = planes.shape
    if not (0 < groups <= 255 and 0 < out_features <= 65536):
        raise RuntimeError("dimensions outside v1 bounds")
    if out_features % 32:
        raise RuntimeError("v1 requires O divisible by 32 for aligned plane rows")
    if x.shape[1] != groups * 128:
        raise RuntimeError("K mismatch")
    if scales.dtype not in (torch.bfloat16, torch.float16) or tuple(scales.shape) != (groups, out_features):
        raise RuntimeError("deployment scales must be BF16 [G,O]")
    if perm.dtype != torch.int16 or perm.ndim != 1 or perm.numel() != groups * 128:
        raise RuntimeError("perm must be int16 [K]")
    if partial.dtype != torch.float32 or tuple(partial.shape) != (splits, out_features):
        raise RuntimeError("partial has wrong FP32 [splits,O] shape")


def workspace_shape(out_features: int, in_features: int, groups_per_split: int = 1) -> tuple[int, int]:
    """Shape of the caller-owned FP32 workspace: one row per K split, ``O`` columns."""
    if not 1 <= out_features <= 65536 or not 128 <= in_features <= 32767 or in_features % 128:
        raise ValueError("invalid W3 LUT dimensions")
    groups = in_features // 128
    if not isinstance(groups_per_split, int) or not 1 <= groups_per_split <= groups:
        raise ValueError("groups_per_split must be an integer in [1,K/128]")
    return -(-groups // groups_per_split), out_features


def _layout_args(layout, wait=True):
    return layout["planes"], layout["scales"], layout.get("zeros"), _perm_or_none(layout["perm"], wait)


class _LayoutRecord:
    """A validated layout and the launches prepared for it.  Holds no tensor: it goes when the planes go."""

    __slots__ = ("out_features", "in_features", "index", "seen", "launches", "recent", "keeper")

    def __init__(self, layout):
        self.out_features, self.in_features = validate_planar_w3(layout, check_values=False)
        # what the checks looked at, so that they hold only while it does; the perm with its version: a launch knows whether it
        # was the identity
        self.seen = tuple((name, weakref.ref(value), _native.calls().stamp(value, name == "perm")) for name, value in layout.items())
        self.index, self.launches, self.recent = layout["planes"].get_device(), {}, None


_RECORDS: dict[int, _LayoutRecord] = {}


def _layout_record(layout) -> _LayoutRecord:
    planes = layout.get("planes")
    key = id(planes)
    record = _RECORDS.get(key)
    if record is None or not _native.calls().holds(layout, record.seen):
        record = _LayoutRecord(layout)
        record.keeper = weakref.ref(planes, lambda _: _RECORDS.pop(key, None))
        _RECORDS[key] = record
    return record


def _launch_layout(record, layout, x, out, kind, decoded) -> None:
    if x.get_device() != record.index:
        raise ValueError("x, out and the layout must share a device")
    if not (x.is_contiguous() and out.is_contiguous()):  # the kernels know rows that lie side by side only
        packed = torch.empty(out.shape, device=out.device, dtype=out.dtype)
        _launch_layout(record, layout, x.contiguous(), packed, kind, decoded)
        out.copy_(packed)
        return
    key = (kind, x.shape[0], x.dtype, decoded)
    launch = record.launches.get(key, 0)
    if not launch:
        # a first call, or a column order that cannot be looked at now: the plain entry points.  The second
        # call prepares the launch (about 40 us), which pays from a few calls on.
        prepare = launch is None and not torch.cuda.is_current_stream_capturing()
        if launch == 0:
            record.launches[key] = None
        elif prepare:
            record.launches[key] = _native.Launch(kind, x.dtype, _layout_args(layout), record.out_features, record.in_features,
                                                  rows=x.shape[0], decoded=decoded, hold=False)
        planes, scales, zeros, perm = _layout_args(layout, wait=False)
        if kind == "small":
            _native.w3_gemm_small(x, planes, scales, zeros, perm, out)
        else:
            _native.w3_gemv(x, planes, scales, zeros, perm, out, decoded_bf16=decoded)
        return
    launch.call.run(x, out)


def inline_main(x, layout, workspace, *, row_tile: int, arithmetic: str = "structural") -> None:
    """First half of the two-call form: ``workspace[g, o]`` receives group ``g``'s scaled sum."""
    out_features, in_features = validate_planar_w3(layout, check_values=False)
    if x.shape != (1, in_features):
        raise ValueError("x must have shape [1,K]")
    if arithmetic not in ARITHMETIC_MODES:
        raise ValueError(f"arithmetic must be one of {ARITHMETIC_MODES}")
    if workspace.shape != workspace_shape(out_features, in_features) or workspace.dtype != torch.float32:
        raise ValueError("workspace must be FP32 [K/128,O]")
    if workspace.device != x.device or any(value.device != x.device for value in layout.values()):
        raise ValueError("x, layout and workspace must share a device")
    load_w3_lut_extension(row_tile)
    planes, scales, zeros, perm = _layout_args(layout)
    _native.w3_gemv(x, planes, scales, zeros, perm, workspace,
                    decoded_bf16=arithmetic == "decoded_bf16", group_partials=True)


def finish(workspace, out, *, row_tile: int):
    """Second half: ``out[0, o] = sum_g workspace[g, o]`` in ascending group order."""
    if workspace.ndim != 2 or workspace.dtype != torch.float32:
        raise ValueError("workspace must be FP32 [G,O]")
    if out.shape != (1, workspace.shape[1]) or out.dtype not in (torch.float16, torch.bfloat16):
        raise ValueError("out must be FP16/BF16 [1,O]")
    load_w3_lut_extension(row_tile).finish(workspace, out)
    return out


def w3_lut_m1_out(x, layout, out, workspace, *, row_tile: int, groups_per_split: int = 1,
                  arithmetic: str = "structural"):
    """Allocation-free M=1 GEMV on the current CUDA stream; returns ``out``.

    ``workspace`` must have the reference's shape for ``groups_per_split`` but is not
    written: the K split is reduced inside the kernel through a small per-stream scratch.
    """
    if out.dtype != x.dtype:
        raise ValueError("out dtype must match x dtype")
    if arithmetic not in ARITHMETIC_MODES:
        raise ValueError(f"arithmetic must be one of {ARITHMETIC_MODES}")
    record = _layout_record(layout)
    out_features, in_features = record.out_features, record.in_features
    if x.shape != (1, in_features) or out.shape != (1, out_features):
        raise ValueError("x/out shape mismatch")
    if workspace.shape != workspace_shape(out_features, in_features, groups_per_split) or workspace.dtype != torch.float32:
        raise ValueError("workspace must be FP32 [ceil(G/groups_per_split),O]")
    if workspace.device != x.device or out.device != x.device:
        raise ValueError("x, out and workspace must share a device")
    load_w3_lut_extension(row_tile)
    _launch_layout(record, layout, x, out, "w3", arithmetic == "decoded_bf16")
    return out


def w3_lut_gemv_out(x, layout, out, *, arithmetic: str = "structural", kernel: str = "auto"):
    """Small-batch form (``x`` is ``[M,K]``, M = 1..16) of ``w3_lut_m1_out``; no reference counterpart.

    ``kernel``: ``"lut"`` is the table-lookup kernel (M <= 4, cost grows with M), ``"mma"`` the
    tensor-core kernel (M <= 16, cost hardly grows with M; weights are not rounded).  ``"auto"`` picks
    ``"lut"`` for one row (4096 x 4096: 3.8 us against 5.1) and for the dequantised-weight arithmetic, which
    only that kernel has, and ``"mma"`` from two rows on (two rows: 5.1 us against 5.6, four: 5.3 against 9.3).
    """
    record = _layout_record(layout)
    recent = record.recent
    if recent is not None and recent[0] == kernel and recent[1] == arithmetic and recent[2](x, out):  # the operands fit that launch
        return out
    rows = x.shape[0] if x.ndim else 0
    if x.ndim != 2 or x.shape[1] != record.in_features or out.shape != (rows, record.out_features):
        raise ValueError("x/out shape mismatch")
    if out.dtype != x.dtype or out.device != x.device:
        raise ValueError("out must match x in dtype and device")
    asked = kernel
    if kernel == "auto":
        kernel = "lut" if rows == 1 or arithmetic == "decoded_bf16" else "mma"
    elif kernel not in ("lut", "mma"):
        raise ValueError("kernel must be auto, lut or mma")
    if rows < 1 or rows > (4 if kernel == "lut" else 16):
        raise ValueError(f"the {kernel} kernel takes 1..{4 if kernel == 'lut' else 16} rows")
    if kernel == "mma" and arithmetic != "structural":
        raise ValueError("the tensor-core kernel has one arithmetic: weights that are not rounded")
    kind, decoded = "small" if kernel == "mma" else "w3", arithmetic == "decoded_bf16"
    _launch_layout(record, layout, x, out, kind, decoded)
    launch = record.launches.get((kind, rows, x.dtype, decoded))
    if launch:
        record.recent = (asked, arithmetic, launch.call.fits)
    return out


def dense_linear(x, layout, bias=None):
    """``x`` ``[T,K]`` (16-bit, CUDA) times the dequantised weight, without the packed kernels' row limit: up to 16 rows
    without a bias stay packed (the tensor-core kernel, whose weights are not rounded at all), the rest, its
    activations gathered into group-sorted column order, goes through the kernel that dequantises into tensor memory or
    through dense chunks of the weight."""
    planes, scales, zeros, perm = _layout_args(layout)
    rows, (out_features, in_features) = x.shape[0], (planes.shape[2], x.shape[1])
    y = torch.empty(rows, out_features, device=x.device, dtype=x.dtype)
    x = x.contiguous()
    # a bias added to the packed kernel's rounded output would round twice
    if rows <= 16 and bias is None and out_features % 32 == 0 and x.data_ptr() % 16 == 0:
        _native.w3_gemm_small(x, planes, scales, zeros, perm, y)
        return y
    if perm is not None:
        ordered = torch.empty_like(x)
        _native.gather_columns(x, perm, ordered)
        x = ordered
    if fused_gemm_pays(rows, out_features) and x.data_ptr() % 16 == 0:
        _native.w3_gemm(x, (layout,), y, None if bias is None else bias.to(x.dtype).expand(rows, out_features).contiguous())
        return y
    chunks = -(-out_features * in_features * 2 // DENSE_CHUNK_BYTES)
    step = -(-(-(-out_features // chunks)) // 64) * 64
    weight = torch.empty(min(step, out_features), in_features, device=x.device, dtype=x.dtype)
    for begin in range(0, out_features, step):
        count = min(step, out_features - begin)
        _native.w3_dequant([(layout, weight)], x.dtype, row_begin=begin, row_count=count)
        target = y[:, begin:begin + count]
        if bias is None:
            torch.mm(x, weight[:count].t(), out=target)
        elif count == out_features:
            torch.addmm(bias, x, weight.t(), out=y)
        else:  # into columns of a wider output the library rounds the product before it adds (error 2.3e-3 against 1.7e-3)
            target.copy_(F.linear(x, weight[:count], bias[begin:begin + count]))
    return y


def qwen3_row_tile(out_features: int, in_features: int) -> int:
    try:
        return QWEN3_ROW_TILE_BY_SHAPE[(out_features, in_features)]
    except KeyError as exc:
        raise ValueError(f"unsupported Qwen3-8B W3 shape: {(out_features, in_features)}") from exc


def qwen3_w3_route(route: str, out_features: int, in_features: int) -> dict:
    if route not in QWEN3_W3_ROUTE_POLICIES:
        raise ValueError(f"unknown Qwen3-8B W3 route: {route}")
    try:
        return dict(QWEN3_W3_ROUTE_POLICIES[route][(out_features, in_features)])
    except KeyError as exc:
        raise ValueError(f"unsupported Qwen3-8B W3 shape: {(out_features, in_features)}") from exc


class PackedW3Linear(nn.Module):
    """Decode-only W3 ``Linear``: packed GEMV for one token, explicit dense fallback otherwise.

    Construction clones the layout into buffers.  A bound ("prepared") module owns one
    reusable ``[1,O]`` output and returns a view of it on every call, so a consumer must
    finish with it, on the same stream, before the next call; use is serial and batch-one,
    which is what a whole-sequence CUDA graph needs (no allocation per call).
    """

    def __init__(self, layout, *, bias=None, fallback: str = "error", row_tile: int | None = None,
                 groups_per_split: int = 1, arithmetic: str = "structural", route: str = "structural"):
        super().__init__()
        if fallback not in {"error", "dense"}:
            raise ValueError("fallback must be error or dense")
        self.out_features, self.in_features = validate_planar_w3(layout)
        self.row_tile = qwen3_row_tile(self.out_features, self.in_features) if row_tile is None else row_tile
        if self.row_tile not in ROW_TILES:
            raise ValueError(f"row_tile must be one of {ROW_TILES}")
        if arithmetic not in ARITHMETIC_MODES:
            raise ValueError(f"arithmetic must be one of {ARITHMETIC_MODES}")
        if arithmetic == "decoded_bf16" and "zeros" in layout:
            # the kernel's rounding correction covers code - zero = +/-3, the only inexact
            # products at zero points 3 and 4; other zero points have further inexact products
            zero_values = set(torch.unique(layout["zeros"]).tolist())
            if not zero_values <= {3, 4}:
                raise ValueError("decoded_bf16 arithmetic needs zero points 3 or 4")
        workspace_shape(self.out_features, self.in_features, groups_per_split)
        self.groups_per_split = groups_per_split
        self.arithmetic = arithmetic
        self.route = route
        self.fallback = fallback
        self.route_counts = {"packed_m1": 0, "dense_fallback": 0}
        self.last_route = "not_called"
        self._decode_binding = None
        self._decode_audit = False
        self._valid_values = None
        self._fields = tuple(name for name in FIELDS + OPTIONAL_FIELDS if name in layout)
        for name in self._fields:
            self.register_buffer(name, layout[name].detach().clone())
        self.register_buffer("bias", None if bias is None else bias.detach().clone())
        self.register_buffer("_workspace", None, persistent=False)
        self.register_buffer("_decode_output", None, persistent=False)

    def layout(self) -> dict[str, torch.Tensor]:
        return {name: getattr(self, name) for name in self._fields}

    def _require_valid_values(self, layout) -> None:
        """The value checks of ``validate_planar_w3`` (they synchronise), once per state of the buffers: these very tensors, where
        they were, not written to since (inference tensors do not tell, and are checked every time)."""
        seen = self._valid_values
        if seen is None or len(seen) != len(layout) or any(owner() is not t or address != t.data_ptr() or version != t._version
                                                           for (owner, address, version), t in zip(seen, layout.values())):
            validate_planar_w3(layout)
            known = not any(t.is_inference() for t in layout.values())
            self._valid_values = tuple((weakref.ref(t), t.data_ptr(), t._version) for t in layout.values()) if known else None

    def __getstate__(self):
        return {**self.__dict__, "_valid_values": None}  # weak references, to the buffers of this module

    def clear_prepared_decode(self) -> None:
        self._decode_binding = None
        self._decode_output = None
        self._workspace = None
        self._decode_audit = False

    def _apply(self, fn, recurse=True):
        # any device / dtype move invalidates the tensors a binding captured
        self.clear_prepared_decode()
        return super()._apply(fn, recurse=recurse)

    def bind_prepared_decode(self, dtype: torch.dtype) -> None:
        if self._decode_binding is not None:
            raise ValueError("decode already bound")
        if dtype not in (torch.float16, torch.bfloat16):
            raise ValueError("FP16/BF16 required")
        layout = self.layout()
        device = layout["planes"].device
        if device.type != "cuda":
            raise ValueError("prepared decode requires CUDA")
        validate_planar_w3(layout, check_values=False)
        load_w3_lut_extension(self.row_tile)
        planes, scales, zeros, perm = _layout_args(layout)
        corrected = self.arithmetic == "decoded_bf16"
        # The reference's workspace is kept (same shape contract) although the kernel does
        # not need it; the shared per-stream scratch is sized here, before any capture.
        self._workspace = torch.empty(
            workspace_shape(self.out_features, self.in_features, self.groups_per_split),
            device=device, dtype=torch.float32)
        _native.scratch_for(device, _native.w3_scratch_bytes(1, self.out_features, self.in_features))
        self._decode_output = torch.empty((1, self.out_features), device=device, dtype=dtype)
        output = self._decode_output
        shaped = output.view(1, 1, self.out_features)
        launch = _native.Launch("w3", dtype, (planes, scales, zeros, perm), self.out_features, self.in_features, decoded=corrected)
        # a weak reference to the module, so no cycle: a dropped module gives its weights back at once
        self._decode_binding = _native.calls().Bound(launch.call, launch, output, shaped, weakref.ref(self), self._buffers)

    def _launches(self, x, rows) -> bool:
        """Whether the dense fallback may go through the kernels; what they do not take, and what tensor operations refuse
        (a bias of another dtype), is left to tensor operations."""
        return (x.is_cuda and x.dtype in (torch.float16, torch.bfloat16) and x.device == self.planes.device and rows > 0
                and (self.bias is None or (self.bias.dtype == x.dtype and self.bias.device == x.device and self.bias.shape == (self.out_features,)))
                and _native.plain_tensors(x, self.bias, *self.layout().values()) and self.planes.data_ptr() % 16 == 0 and self.perm.data_ptr() % 16 == 0)

    def adds_residual(self, x: torch.Tensor) -> bool:
        """Whether ``add_to`` can stand for a call of this bound module and an addition."""
        return (self._decode_binding is not None and self.bias is None and self._decode_output.dtype == x.dtype and x.is_cuda and x.is_contiguous()
                and x.numel() == self.in_features and x.get_device() == self._decode_output.get_device())

    def add_to(self, residual: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
        """``residual + self(x)`` for one token in one launch, with the roundings of the two steps."""
        if self._decode_audit:
            self.route_counts["packed_m1"] += 1
            self.last_route = "packed_m1"
        planes, scales, zeros, perm = _layout_args(self.layout(), wait=False)
        out = torch.empty_like(residual)
        _native.w3_gemv_multi(x.view(1, self.in_features), _native.w3_matrix_list([(planes, scales, zeros, out, residual)]), 1, self.out_features, scales.dtype,
                              perm, decoded_bf16=self.arithmetic == "decoded_bf16")
        return out

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if self._decode_binding is not None:
            return self._decode_binding(x)
        if torch.is_grad_enabled():
            raise RuntimeError("packed inference requires no_grad/inference_mode")
        if x.ndim < 2 or x.shape[-1] != self.in_features:
            raise ValueError("expected [...,K] input")
        layout = self.layout()
        rows = x.numel() // self.in_features
        if rows != 1 or not x.is_cuda or x.dtype not in (torch.float16, torch.bfloat16):
            if self.fallback != "dense":
                raise ValueError("unsupported input; enable explicit dense fallback if needed")
            self.last_route = "dense_fallback"
            self.route_counts["dense_fallback"] += 1
            if not self._launches(x, rows):
                return F.linear(x, restore_planar_w3(layout, dtype=x.dtype), self.bias)
            self._require_valid_values(layout)
            return dense_linear(x.reshape(rows, self.in_features), layout, self.bias).reshape(*x.shape[:-1], self.out_features)
        self.last_route = "packed_m1"
        self.route_counts["packed_m1"] += 1
        shape = workspace_shape(self.out_features, self.in_features, self.groups_per_split)
        if self._workspace is None or self._workspace.device != x.device or tuple(self._workspace.shape) != shape:
            self._workspace = torch.empty(shape, device=x.device, dtype=torch.float32)
        output = torch.empty((1, self.out_features), device=x.device, dtype=x.dtype)
        w3_lut_m1_out(x.reshape(1, self.in_features).contiguous(), layout, output, self._workspace,
                      row_tile=self.row_tile, groups_per_split=self.groups_per_split, arithmetic=self.arithmetic)
        if self.bias is not None:
            output.add_(self.bias)
        return output.reshape(*x.shape[:-1], self.out_features)


def replace_w3_block_linears(block, layer_payload, *, fallback: str = "error",
                             row_tile_by_shape: dict[tuple[int, int], int] | None = None,
                             route: str = "structural") -> list[str]:
    """Swap the seven Linears of one Qwen3 decoder block; nothing is touched unless all seven validate."""
    from .qwen3 import QWEN3_LINEAR_MODULES

    fields_of = lambda name: [f for f in FIELDS + OPTIONAL_FIELDS if f"{name}.{f}" in layer_payload]  # noqa: E731
    required = {f"{module}.{field}" for module in QWEN3_LINEAR_MODULES for field in FIELDS}
    allowed = required | {f"{module}.{field}" for module in QWEN3_LINEAR_MODULES for field in OPTIONAL_FIELDS}
    if not required <= set(layer_payload) or not set(layer_payload) <= allowed:
        raise ValueError("layer must contain exactly seven complete W3 payloads")
    if route not in QWEN3_W3_ROUTE_POLICIES:
        raise ValueError(f"unknown Qwen3-8B W3 route: {route}")
    tiles = QWEN3_ROW_TILE_BY_SHAPE if row_tile_by_shape is None else row_tile_by_shape
    staged = []
    for name in QWEN3_LINEAR_MODULES:
        old = block.get_submodule(name)
        layout = {field: layer_payload[f"{name}.{field}"] for field in fields_of(name)}
        shape = validate_planar_w3(layout)
        if not isinstance(old, nn.Linear) or (old.out_features, old.in_features) != shape:
            raise ValueError(f"Linear shape/type mismatch: {name}")
        if shape not in tiles:
            raise ValueError(f"row-tile policy missing shape: {shape}")
        tile = tiles[shape]
        if row_tile_by_shape is None:
            policy = qwen3_w3_route(route, *shape)
            if policy["row_tile"] != tile:
                raise ValueError("route and row-tile policies disagree")
        else:
            policy = {"groups_per_split": 1, "arithmetic": "structural"}
        module = PackedW3Linear(layout, bias=old.bias, fallback=fallback, row_tile=tile,
                                groups_per_split=policy["groups_per_split"],
                                arithmetic=policy["arithmetic"], route=route).to(old.weight.device)
        staged.append((name, module))
    for name, module in staged:
        parent, attribute = name.rsplit(".", 1)
        setattr(block.get_submodule(parent), attribute, module)
    return [name for name, _ in staged]
