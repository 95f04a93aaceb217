"""Planes read through the staging buffer: one larger than the buffer (64 MB)
equals its two halves, ghost columns included."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("precision", [0, 1])
def test_plane_larger_than_the_staging_buffer(iris, tmp_path, precision):
    nx, ny, nz = 1401, 1003, 13
    w = cfg.Workload("plane", nx, ny, nz, 3, 11, 6, 1, 2.25, 0, 5, (1, nx, 1, ny, 4, 10), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=2))
    p.akx_re, p.aky_re, p.dft_faces = 0.3, 0.2, iris.DFT_Z
    e = iris.Engine(p, fw, precision=precision, dft_block=4)
    e.step(150, 3)
    a = e.get_plane(iris.E, 3, 5, (0, nx + 1), (0, ny + 1))
    lo = e.get_plane(iris.E, 3, 5, (0, nx + 1), (0, 500))
    hi = e.get_plane(iris.E, 3, 5, (0, nx + 1), (501, ny + 1))
    assert a.nbytes > 64 << 20 and np.any(a)
    assert np.array_equal(a, np.concatenate([lo, hi]))
    y = e.get_plane(iris.E, 2, 501, (0, nx + 1), (0, nz + 1))
    assert np.array_equal(y[5], a[501])
    e.close()
