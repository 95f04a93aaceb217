"""Grids with more rows or planes than 65535 tiles: what a launch maps to grid.y or
grid.z must still fit.  A column of cells long in y (the TF/SF corrections of
unsampled steps are a launch of their own) against the persistent kernel, whose
launch does not depend on the grid's shape."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


def workload(iris, tmp_path, nx, ny, nz, pml, zi, nof=2):
    w = cfg.Workload("long", nx, ny, nz, pml, nz + 1 - pml, pml + 2, 2, 2.25, 0, zi, (1, nx, 1, ny, pml + 1, nz - pml), nof, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=1 if nx == 1 else 2, sample_fourier=4))
    p.dft_faces = iris.DFT_Z
    return p, fw


@pytest.mark.parametrize("precision", [0, 1])
def test_rows_past_65535_correction_tiles(iris, tmp_path, precision):
    p, fw = workload(iris, tmp_path, 1, 263000, 8, 2, 4)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_PERSISTENT, iris.STENCIL_DEFAULT):
        e = iris.Engine(p, fw, precision=precision, stencil=st)
        e.step(150, 7)
        e.tfsf(160)
        e.sync()
        out.append([e.get_plane(f, 1, 1, (0, p.ny + 1), (0, p.nz + 1)) for f in (iris.E, iris.H)] + [e.flux(0)])
        e.close()
    assert np.any(out[0][0][4, 262900:]) and np.any(out[0][2])
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("ny,form", [(327000, 1), (328000, 0)])
def test_rows_past_65535_slab_tiles(iris, tmp_path, ny, form):
    """The fused pass with its tiles, five rows high in the slabs, filling grid.y and
    with the unstaged column where they no longer fit, against the split passes."""
    p, fw = workload(iris, tmp_path, 40, ny, 9, 2, 4)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_FUSED):
        e = iris.Engine(p, fw, precision=iris.FP32, stencil=st)
        if st == iris.STENCIL_FUSED:
            assert e.stepping()["form"] == form
        e.material_pattern(3, 0.5)
        e.step(150, 5)
        out.append([e.get_plane(f, 1, 17, (0, p.ny), (1, p.nz)) for f in (iris.E, iris.H)] +
                   [e.get_plane(iris.E, 2, p.ny, (1, p.nx), (1, p.nz)), e.flux(0)])
        e.close()
    assert np.any(out[0][0][:, 326900:]) and np.any(out[0][3])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_planes_past_65535_chunks(iris, tmp_path):
    """A source near z = 1: what passes the slab there comes back at the last planes,
    across the period in z."""
    p, fw = workload(iris, tmp_path, 2, 3, 930000, 4, 8)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_FUSED):
        e = iris.Engine(p, fw, precision=iris.FP32, stencil=st)
        e.step(150, 40)
        out.append([e.get_plane(f, 2, 2, (1, 2), r) for f in (iris.E, iris.H) for r in ((1, 60), (929940, p.nz))] + [e.flux(0)])
        e.close()
    assert np.any(out[0][0]) and np.any(out[0][1][929985 - 929940])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
