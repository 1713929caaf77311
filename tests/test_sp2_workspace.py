"""The workspace of the SCF loops' purification covers what its one launch addresses, at every size the launch takes.  No GPU."""
import ctypes

from rerdmft_b200 import _lib


def test_workspace_covers_the_one_launch_purification():
    lib, have, need = _lib.lib(), ctypes.c_int64(), ctypes.c_int64()
    for cplx in (0, 1):
        sizes = 0
        for n in range(1, 520):
            assert lib.rr_test_sp2_workspace(n, cplx, ctypes.byref(have), ctypes.byref(need)) == _lib.RR_OK
            assert have.value >= need.value, (n, cplx, have.value, need.value)
            sizes += need.value > 0
        assert sizes >= 400
