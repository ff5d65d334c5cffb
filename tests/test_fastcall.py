"""The call binding of the C ABI: every argument kind arrives as ctypes would pass it, and what it does not take goes to ctypes."""
import ctypes as C
import platform
import subprocess

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


def test_what_ctypes_refuses_is_refused():
    """Handles of another kind, arrays of another type and numbers where a typed pointer is due."""
    L = abi.lib()
    S, segs = abi.StreamWrapper(0), (abi.Segment * 1)()
    clear = lambda seg: L.zg_segment_sumsq(9, S, None, seg, 1, None)
    for seg in (segs, None):
        L.zg_clear_error()
        clear(seg)
        assert L.zg_last_error() == 5  # called: an unsupported dtype
    L.zg_clear_error()
    for bad in (64, b"12345678", (abi.len_t * 2)(), (abi.Block * 1)(), "x"):
        with pytest.raises((TypeError, C.ArgumentError)):
            clear(bad)
    for bad in (abi.CublasWrapper(0), abi.GraphWrapper(0), abi.Block(0, 0), 64, None):
        with pytest.raises((TypeError, C.ArgumentError)):
            L.stream_synchronize(bad)
    assert L.zg_last_error() == 0


def test_bool_arguments_are_one_or_zero(tmp_path):
    src = tmp_path / "f.c"
    src.write_text("unsigned long f(unsigned long a, unsigned long b) { return a * 1000 + b; }")
    subprocess.run(["gcc", "-shared", "-fPIC", str(src), "-o", str(tmp_path / "f.so")], check=True)
    fn = C.CDLL(str(tmp_path / "f.so")).f
    abi.lib()
    g = abi._fast.function(C.cast(fn, C.c_void_p).value, "bi", "u", fn, (None, None))
    assert [g(x, 7) for x in (True, False, 1, 0, 2, -4, 1 << 40)] == [1007, 7, 1007, 7, 1007, 1007, 1007]
