"""pb_hierarchy_setup_f32 makes level 0 from its screen, so it refuses to go without one
(pb_hierarchy_setup_sparse_f32 takes level 0's arrays as they are).  No GPU: arguments are
checked before any device work."""

import ctypes


def test_null_screen_is_refused():
    from mojo_poissonrecon_b200 import _native

    L = _native.lib()
    sides = (ctypes.c_int64 * 2)(5, 3)
    arrays = (ctypes.c_void_p * 16)(*[16] * 16)  # never dereferenced
    status = L.pb_hierarchy_setup_f32(2, sides, arrays, 0, None, 4.0, 16, 0, 16, 16, 0, None)
    assert status == 1, status  # PB_ERR_INVALID
    assert "screen" in L.pb_last_error().decode()
