"""The build on other hosts, and what was built for another torch or another Python: neither taken for up to date nor used."""
import ctypes
import shutil
import subprocess

import pytest
import torch

from marlin_style_fluxbin_b200 import _native, build


def test_the_fingerprint_follows_torch_and_the_python_abi(monkeypatch):
    before = build._fingerprint()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build._fingerprint() != before
    monkeypatch.undo()
    assert build._fingerprint() == before
    monkeypatch.setattr(build, "CALLS", build.CALLS.with_name("_fb_calls.cpython-399-x86_64-linux-gnu.so"))
    assert build._fingerprint() != before


def test_a_module_for_another_torch_is_refused_with_the_reason(monkeypatch):
    if _native._calls is None:
        pytest.skip("not built")
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    module, error = _native._load_calls()
    assert module is None and "0.0.1" in str(error)
    monkeypatch.undo()
    monkeypatch.setattr(_native, "_calls", None)
    monkeypatch.setattr(_native, "_calls_error", ImportError("undefined symbol: nowhere"))
    with pytest.raises(RuntimeError, match="undefined symbol: nowhere") as caught:
        _native.calls()
    assert isinstance(caught.value.__cause__, ImportError)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_the_portable_host_code_packs_the_same_planes(tmp_path):
    """What a host without x86 instructions runs, against the tensor form; 80 columns: a block of 64 and a partial one."""
    from marlin_style_fluxbin_b200.gptq_deployment import planes_from_sorted_codes, unpack_gptq_w3_qweight

    stub = tmp_path / "stub.cpp"
    stub.write_text("namespace fb { int fail(int code, const char*, ...) { return code; } }")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-DFB_PORTABLE", str(build.CSRC / "fb_host_pack.cpp"), str(stub), "-o", str(tmp_path / "pack.so"),
                    "-lpthread"], check=True)
    lib = ctypes.CDLL(str(tmp_path / "pack.so"))
    gen = torch.Generator().manual_seed(1)
    words = torch.randint(-2**31, 2**31, (24, 80), dtype=torch.int64, generator=gen).to(torch.int32)
    order, planes = torch.randperm(256, generator=gen), torch.empty(2, 3, 80, 16, dtype=torch.uint8)
    pointer = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.fb_host_w3_planes(pointer(words), pointer(order), 256, 80, pointer(planes), 2) == 0
    assert torch.equal(planes, planes_from_sorted_codes(unpack_gptq_w3_qweight(words)[order]))
