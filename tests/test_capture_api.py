"""tg_capture_own and tg_capture_release refuse what no capture stands behind,
before they touch CUDA."""
import ctypes


def test_refusals_without_a_device(pkg):
    L = pkg.colsolve.lib()
    assert L.tg_capture_own(None, None) == pkg.TG_EINVAL
    assert L.tg_capture_release(ctypes.c_ulonglong(5)) == pkg.TG_EINVAL
