"""The host-side extension is an accelerator: where it is missing or cannot be built, calls go through the Python path."""
import warnings

import pytest

from flash_pop_b200 import _lib


@pytest.fixture
def unloaded(monkeypatch):
    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.setattr(_lib, "_native_bound", None)


@pytest.mark.parametrize("content", [None, b"not a shared object"])
def test_a_missing_or_unloadable_extension_declines(unloaded, monkeypatch, tmp_path, content):
    path = tmp_path / "fpb_fast_calls.so"
    if content is not None:
        path.write_bytes(content)
    _lib.build()
    monkeypatch.setattr(_lib, "_native_path", lambda: str(path))
    with pytest.warns(UserWarning, match="no host-side extension"):
        native = _lib.native()
    with warnings.catch_warnings():
        warnings.simplefilter("error")               # (says so once)
        assert _lib.native() is native
    assert native.forward(1, 2, 3) is None and native.column_sums(None, None) is None
    assert _lib.result(native.step()) is None


@pytest.mark.parametrize("command", [["/nonexistent/g++"], ["false"]])
def test_build_goes_on_without_a_host_compiler(monkeypatch, command):
    _lib.build()
    monkeypatch.setattr(_lib, "_native_command", lambda out: command)
    monkeypatch.setattr(_lib, "_native_stale", lambda: True)
    with pytest.warns(UserWarning, match="host-side extension"):
        assert _lib.build() == _lib.LIB_PATH
