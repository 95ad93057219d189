"""A kernel that copies planes by tensor maps is not launched where a map cannot
be made (its copies would read wherever the unset map's bytes say): the
launchers return without a launch and mark the context, in every precision."""
import ctypes as C

import pytest


@pytest.mark.parametrize("precision", [64, 65, 32])
def test_no_launch_without_a_map(built, precision):
    from lare3d_b200 import gpu
    f = gpu.library().lare_gpu_check_unmapped
    f.argtypes = [C.c_int, C.POINTER(C.c_longlong)]
    n = C.c_longlong(-1)
    assert f(precision, C.byref(n)) == -2  # LARE_ECUDA
    assert n.value == 0


def test_check_arguments(built):
    from lare3d_b200 import gpu
    f = gpu.library().lare_gpu_check_unmapped
    f.argtypes = [C.c_int, C.POINTER(C.c_longlong)]
    assert f(64, None) == -1 and f(16, C.byref(C.c_longlong())) == -1
