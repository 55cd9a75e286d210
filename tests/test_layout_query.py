"""pwmgpu_layout's argument checks, without a GPU."""
import ctypes


def test_layout_rejects_bad_arguments():
    import thesis_spmv_gb300 as t
    L, k = t.lib(), ctypes.c_int32()
    assert L.pwmgpu_layout(None, 0, ctypes.byref(k)) == 1  # PWMGPU_ERR_INVALID
