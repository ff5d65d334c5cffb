"""The call binding of the C ABI: every argument kind arrives as ctypes would pass it, and what it does not take goes to ctypes."""
import ctypes as C

import pytest

from zigrad_b200 import abi


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
