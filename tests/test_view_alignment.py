"""CPU: a batch stride that is no whole number of elements is refused on the host.  The
kernels address images by byte strides, so every image but the first would be read
and written at misaligned addresses.  A single image's stride is not used."""
import ctypes as C

import pytest


@pytest.mark.parametrize("dtype,es", [("F32", 4), ("BF16", 2), ("U8X4", 4)])
def test_misaligned_batch_stride_is_refused(hgb_lib, dtype, es):
    from hipacc_gb300 import _lib as L

    def view(batch, stride):
        return L.View(0x1000, getattr(L, dtype), 16, 16, batch, 16 * es, stride)

    bad, good = view(2, 256 * es + 1), view(2, 256 * es)
    m = (C.c_float * 15)()
    if dtype == "U8X4":
        rc = hgb_lib.hgb_unsharp(C.byref(bad), C.byref(bad), 1, 0, None)
        assert rc == L.ERR_INVALID and b"batch stride" in hgb_lib.hgb_last_error()
        return
    for x, y in ((bad, good), (good, bad)):
        rc = hgb_lib.hgb_local_op(C.byref(x), None, C.byref(y), None, m, None, None, 3, 3, 0, 1, 0.0, None)
        assert rc == L.ERR_INVALID and b"batch stride" in hgb_lib.hgb_last_error()
    if dtype == "F32":
        for mw, mh in ((3, 3), (3, 1), (1, 5)):
            rc = hgb_lib.hgb_local_op_adjoint(None, C.byref(bad), C.byref(good), m, None, mw, mh, 1, None, None)
            assert rc == L.ERR_INVALID and b"batch stride" in hgb_lib.hgb_last_error()
        rc = hgb_lib.hgb_separable_adjoint(C.byref(bad), C.byref(good), m, m, 5, 1, 0.0, C.byref(good), None, None, None)
        assert rc == L.ERR_INVALID and b"batch stride" in hgb_lib.hgb_last_error()
    # one image: the stride plays no part, the call is refused for its mask alone
    one = view(1, 256 * es + 1)
    rc = hgb_lib.hgb_local_op(C.byref(one), None, C.byref(one), None, m, None, None, 17, 3, 0, 1, 0.0, None)
    assert rc == L.ERR_INVALID and b"mask size" in hgb_lib.hgb_last_error()
