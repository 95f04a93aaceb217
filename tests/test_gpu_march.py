"""The staged z-marching fused pass (FP32): bit for bit the split passes from
random states at the edges of its tile shapes (32x14, 24x19, 16x29, 40x11 and
54x8 cells: one tile exactly, a last tile of one column and one row, odd and
even planes, tiles that touch no border, a plane of one cell, rows of one
column) and of its z chunks (14 to 27 planes), with Bloch phases on every
axis, real and complex material."""
import importlib

import numpy as np
import pytest

from helpers import interior

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")

# nx, ny, planes outside the UPML launch, complex material
CASES = [(32, 14, 13, False), (33, 15, 14, True), (96, 42, 28, False), (24, 19, 15, False), (25, 20, 1, False),
         (16, 29, 2, True), (17, 30, 27, False), (40, 11, 28, False), (41, 12, 29, False), (54, 8, 41, False),
         (55, 9, 3, True), (162, 24, 43, False), (95, 43, 14, True), (1, 1, 28, False), (1, 40, 14, False),
         (40, 1, 14, False), (2, 2, 5, True), (31, 57, 29, True), (161, 25, 16, False)]


@pytest.mark.parametrize("nx,ny,planes,lossy", CASES)
def test_march_equals_split(iris, tmp_path, nx, ny, planes, lossy, pml=4):
    nz = planes + 2 * pml + 1  # the march takes planes pml + 1 .. nz - 1 - pml
    hi, dh = max(pml + 2, nz // 2 - 3), max(1, min(6, planes - 3))
    w = cfg.Workload("march", nx, ny, nz, pml, nz + 1 - pml, hi, dh, 2.25, 0, pml + 1,
                     (1, nx, 1, ny, pml + 1, nz - pml), 5, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=2))
    p.akx_re, p.aky_re, p.akz_re, p.akx_im = 0.3, -0.7, 0.4, 0.05
    r = np.random.default_rng(3)
    shape = (p.hf - p.hi + 3, ny + 2, nx + 2)
    eps = 1.0 / r.uniform(1.0, 6.0, shape) + (1j * r.uniform(-0.02, 0.02, shape) if lossy else 0.0)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_FUSED):
        e = iris.Engine(p, fw, precision=iris.FP32, stencil=st, dft_block=4)
        e.set_material(eps)
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            e.set_field(which, q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape))
            for slab in (0, 1):
                s = e.pml_shape(slab)
                e.set_pml(which, slab, q.normal(size=s) + 1j * q.normal(size=s))
        e.step(150, 6)
        out.append([interior(e.get_field(f), p) for f in (iris.E, iris.H)] +
                   [e.get_pml(f, s) for f in (0, 1) for s in (0, 1)] + [e.flux(0)])
        e.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (k, int(np.sum(a != b)))


def test_march_batch_equals_engines(iris, tmp_path):
    """Cells of every tile shape, more than one launch takes, one without
    planes to march and one with a complex material among real ones."""
    sizes = [(c[0], c[1], 6 + c[2]) for c in CASES] * 3
    sizes[7] = (9, 5, 10)
    ps, mats = [], []
    r = np.random.default_rng(8)
    for c, (nx, ny, nz) in enumerate(sizes):
        w = cfg.Workload("march", nx, ny, nz, 3, 5 if c == 7 else nz - 2, 5, 1, 2.25, 0, 4,
                         (1, nx, 1, ny, 4, 4), 5, 9)
        p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=2))
        p.akx_re, p.aky_re, p.precision = 0.3, -0.7, iris.FP32
        ps.append(p)
        shape = (p.hf - p.hi + 3, ny + 2, nx + 2)
        mats.append(1.0 / r.uniform(1.0, 6.0, shape) + (1j * r.uniform(-0.02, 0.02, shape) if c == 5 else 0.0))
    out = []
    b = iris.Batch(ps, fw, precision=iris.FP32, dft_faces=iris.DFT_Z)
    for c, m in enumerate(mats):
        b.set_material(c, m)
    b.set_tile(7)  # the fused work list
    b.step(150, 7)
    for c, p in enumerate(ps):
        e = iris.Engine(p, fw, precision=iris.FP32, stencil=iris.STENCIL_SPLIT)
        e.set_material(mats[c])
        e.step(150, 7)
        for which in (iris.E, iris.H):
            assert np.array_equal(interior(b.get_field(c, which), p), interior(e.get_field(which), p)), (c, which)
        assert np.any(interior(b.get_field(c, iris.E), p))
        e.close()
    b.close()


@pytest.mark.parametrize("nx,ny,pml,planes,lossy", [(32, 6, 25, 2, False), (33, 7, 13, 6, True), (96, 18, 12, 9, False),
                                                    (24, 9, 24, 3, False), (25, 10, 11, 5, True), (16, 14, 48, 4, False),
                                                    (17, 15, 23, 7, False), (40, 5, 12, 3, True), (121, 16, 30, 2, False),
                                                    (1, 1, 37, 5, False)])
def test_slab_march_equals_split(iris, tmp_path, nx, ny, pml, planes, lossy):
    """The UPML slabs at the edges of their tile shapes (32x6, 24x9, 16x14 and
    40x5) and chunks (12 to 23 planes)."""
    test_march_equals_split(iris, tmp_path, nx, ny, planes, lossy, pml)
