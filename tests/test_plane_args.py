"""iris_get_plane refuses a bad request before it allocates anything for it: the
code is IRIS_EINVAL whatever the range's size, without a device."""
import ctypes

import numpy as np
import pytest


@pytest.mark.parametrize("lo1,hi1,lo2,hi2", [(0, 3, 0, 3), (-2 ** 31, 2 ** 31 - 1, 0, 2 ** 20), (0, 2 ** 31 - 1, 0, 2 ** 31 - 1),
                                             (5, 0, 7, 0)])
def test_bad_plane_is_einval(iris, lo1, hi1, lo2, hi2):
    L = iris.lib()
    a = np.zeros(8)
    d = a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    assert L.iris_get_plane(None, iris.E, 3, 0, lo1, hi1, lo2, hi2, d, d) == -1
    assert L.iris_get_plane_c(None, iris.E, 3, 0, lo1, hi1, lo2, hi2, d) == -1


def test_null_buffers_are_einval(iris):
    assert iris.lib().iris_get_plane(None, iris.E, 3, 0, 0, 1, 0, 1, None, None) == -1


@pytest.mark.gpu
def test_bad_plane_of_an_engine_is_einval(iris, tmp_path):
    import importlib

    cfg = importlib.import_module("irisfdtd-academic_gb300.configs")
    w = cfg.Workload("plane", 5, 4, 30, 3, 28, 12, 4, 2.25, 0, 6, (1, 5, 1, 4, 5, 25), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    e = iris.Engine(p, fw)
    a = np.zeros(3 * 7 * 6)
    d = a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    for args in ((3, 0, -1, 2, 0, 1), (3, 0, 0, 7, 0, 1), (3, 32, 0, 1, 0, 1), (3, 0, 2, 1, 0, 1), (4, 0, 0, 1, 0, 1),
                 (3, 0, -2 ** 31, 2 ** 31 - 1, -2 ** 31, 2 ** 31 - 1)):
        assert e.L.iris_get_plane(e.h, iris.E, *args, d, d) == -1, args
        assert e.L.iris_get_plane_c(e.h, iris.E, *args, d) == -1, args
    assert e.L.iris_get_plane(e.h, iris.E, 3, 6, 0, 6, 0, 5, d, d) == 0
    e.close()
