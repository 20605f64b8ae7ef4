"""What fslbm_step_f32_noalloc says about a corrector order it does not run (checked before any device
is touched; the pointers are never dereferenced)."""
import ctypes

import pytest


@pytest.mark.parametrize("order", [6, 8])
def test_unavailable_order(built, order):
    fn = built.lib().fslbm_step_f32_noalloc
    fn.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 4 + [ctypes.POINTER(built.Params), ctypes.c_double, ctypes.c_void_p]
    prm = built.Params.make(d1=2, blend=0.4, fd_order=order)
    rc = fn(1 << 32, 1 << 33, 1 << 34, 32, 32, 40, 32, ctypes.byref(prm), 0.0, None)
    buf = ctypes.create_string_buffer(256)
    built.lib().fslbm_last_error(buf, 256)
    msg = buf.value.decode()
    # order 6 runs on the pair kernel in a Solve, so no kernel is named as the one it needs
    assert rc == -1 and str(order) in msg and "orders 0/4 only" in msg and "one-column" not in msg
