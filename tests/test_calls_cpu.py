"""Calls of the native library with and without the extension that makes them cheap."""
import ctypes

import pytest

from warpconvnet_b200 import _native
from warpconvnet_b200.csrc import build as csrc_build


def test_the_same_calls_without_the_extension(monkeypatch, tmp_path):
    fast = _native.lib()
    monkeypatch.setattr(_native, "FASTCALL_PATH", str(tmp_path / "_fastcall.so"))
    monkeypatch.setattr(_native, "_lib", None)
    plain = _native.lib()
    assert plain is not fast and plain.wcn_version() == fast.wcn_version()
    for lib in (plain, fast):
        size = ctypes.c_int64(0)
        assert lib.wcn_conv_packed_weight_bytes(0, 27, 64, 64, _native.WCN_F16, ctypes.byref(size)) == 0 and size.value == 27 * 64 * 64 * 2
        before = _native.LAUNCH_COUNTS["wcn_gather_rows"]
        assert lib.wcn_gather_rows(None, 0, None, None, -1, 0, 0, None, None) < 0   # refused, and counted as a call
        assert _native.LAUNCH_COUNTS["wcn_gather_rows"] == before + 1
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            lib.wcn_gather_rows(1)


def test_a_broken_extension_is_left_out(monkeypatch, tmp_path):
    broken = tmp_path / "_fastcall.so"
    broken.write_bytes(b"not a library")
    monkeypatch.setattr(_native, "FASTCALL_PATH", str(broken))
    assert _native._fastcall_bind() is None


def test_the_library_builds_without_a_c_compiler(monkeypatch, tmp_path, capsys):
    monkeypatch.setenv("CC", str(tmp_path / "no-such-compiler"))
    monkeypatch.setattr(csrc_build, "FASTCALL", str(tmp_path / "_fastcall.so"))
    csrc_build.build_fastcall(force=True)
    assert "ctypes" in capsys.readouterr().out
