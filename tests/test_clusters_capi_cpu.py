"""cls_set_clusters / cls_get_clusters reject null arguments without a GPU."""
import ctypes


def test_null_arguments():
    import cls_b200
    lib = cls_b200._capi.load()
    n = ctypes.c_int32()
    assert lib.cls_set_clusters(None, 4, 0) == -1
    assert lib.cls_get_clusters(None, ctypes.byref(n), ctypes.byref(n)) == -1
