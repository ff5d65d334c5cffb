"""The call binding of the C ABI: every argument kind arrives as ctypes would pass it, and what it does not take goes to ctypes."""
import ctypes as C
import platform

import pytest

from zigrad_b200 import abi, build


def test_binding_is_in_place_and_falls_back():
    L = abi.lib()
    assert type(L.zg_bmm).__name__ == "Function" and L.zg_bmm.argtypes[0] is abi.dtype_t
    L.zg_clear_error()
    # 23 integers and pointers and a double, more than the registers hold: an unsupported width, refused before any launch
    L.zg_mlp_tail_fwd_bwd(abi.SINGLE, abi.StreamWrapper(0), 7, 256, 64, 10, *[64] * 6, 0, 10, 1.5, *[64] * 9, 0)
    assert L.zg_last_error() == 5 and b"256 -> 64 -> 10" in L.zg_last_error_message()
    L.zg_clear_error()
    L.zg_clamp_bwd(9, abi.StreamWrapper(0), None, None, None, 3, -1.0, 2)  # an integer where a double is due
    assert L.zg_last_error() == 5 and b"unsupported dtype 9" in L.zg_last_error_message()
    L.zg_clear_error()
    for bad in ((0, "x"), (0,)):
        with pytest.raises((TypeError, C.ArgumentError)):
            L.zg_scatter_add(*bad)
    assert L.zg_mlp_tail_supported(abi.SINGLE, 128, 64, 10) == 1 and L.zg_mlp_tail_supported(abi.DOUBLE, 128, 64, 10) == 0


def test_without_the_binding_ctypes_serves_the_calls(monkeypatch, tmp_path):
    """Hosts that are not x86-64, and interpreters it was not built for."""
    monkeypatch.setattr(abi, "FASTCALL", str(tmp_path / "_fastcall.so"))
    monkeypatch.setattr(platform, "machine", lambda: "aarch64")
    assert not build.build_fastcall(force=True) and not list(tmp_path.iterdir())
    monkeypatch.setattr(abi, "_lib", None)
    L = abi.lib()
    assert type(L.zg_bmm).__name__ == "_FuncPtr" and L.zg_mlp_tail_supported(abi.SINGLE, 128, 64, 10) == 1


def test_binding_belongs_to_one_interpreter(monkeypatch):
    import sysconfig
    assert abi.FASTCALL.endswith(sysconfig.get_config_var("EXT_SUFFIX")) and sysconfig.get_config_var("py_version_nodot") in abi.FASTCALL
