"""What was built for another torch or another Python is neither taken for up to date nor used."""
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
