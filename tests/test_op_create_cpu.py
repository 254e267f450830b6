"""What pt_op_create refuses is what the device has no room for, not a box size."""
import ctypes


def test_no_box_size_is_refused_by_a_rule():
    from pt_b200 import _capi
    lib = _capi.load()
    h = ctypes.c_void_p()
    # larger than any device, so that the allocation fails where there is one
    st = lib.pt_op_create(ctypes.byref(_capi.MeshDesc(2000, 2000, 2000)), ctypes.byref(h))
    assert st != 0 and lib.pt_last_error().startswith(b"pt_op_create: "), lib.pt_last_error()
