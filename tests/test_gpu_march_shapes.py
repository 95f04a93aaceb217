"""Every tile shape of the staged fused pass with tiles that touch no border (three
each way at least), one that is exactly a plane, and ones a cell past it, real and
complex material, in and outside the UPML slabs: bit for bit the split passes
from random states.  The shape that the engine takes is asserted.  (16x29 and,
in the slabs, 16x14 cells are taken on planes of up to two tile columns only, so
all their tiles touch a border.)"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")

# plane, tile and tiles outside the slabs (None: not asserted), the same in them
PLANES = [((96, 42), ((32, 14), (3, 3)), None), ((65, 41), ((32, 14), (3, 3)), None),
          ((72, 57), ((24, 19), (3, 3)), None), ((65, 51), ((24, 19), (3, 3)), None),
          ((132, 30), ((44, 10), (3, 3)), None), ((109, 29), ((44, 10), (3, 3)), None),
          ((162, 24), ((54, 8), (3, 3)), None), ((109, 21), ((54, 8), (3, 3)), None),
          ((16, 29), ((16, 29), (1, 1)), None), ((44, 10), ((44, 10), (1, 1)), None), ((54, 8), ((54, 8), (1, 1)), None),
          ((32, 14), ((32, 14), (1, 1)), None), ((24, 19), ((24, 19), (1, 1)), None), ((45, 11), None, None),
          ((96, 18), None, ((32, 6), (3, 3))), ((81, 16), None, ((32, 6), (3, 3))),
          ((72, 27), None, ((24, 9), (3, 3))), ((65, 26), None, ((24, 9), (3, 3))),
          ((120, 15), None, ((40, 5), (3, 3))), ((82, 15), None, ((40, 5), (3, 3))),
          ((16, 14), None, ((16, 14), (1, 1))), ((40, 5), None, ((40, 5), (1, 1)))]


@pytest.mark.parametrize("lossy", [False, True])
@pytest.mark.parametrize("plane,inside,slab", PLANES)
def test_shape_equals_split(iris, tmp_path, plane, inside, slab, lossy):
    (nx, ny), pml, planes = plane, 13, 15
    nz = planes + 2 * pml + 1
    w = cfg.Workload("shape", nx, ny, nz, pml, nz + 1 - pml, pml + 3, 7, 2.25, 0, pml + 1,
                     (1, nx, 1, ny, pml + 1, nz - pml), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.akx_re, p.aky_re, p.akz_re, p.akx_im, p.dft_faces = 0.3, -0.7, 0.4, 0.05, iris.DFT_Z
    r = np.random.default_rng(3)
    shape = (p.hf - p.hi + 3, ny + 2, nx + 2)
    eps = 1.0 / r.uniform(1.0, 6.0, shape) + (1j * r.uniform(-0.02, 0.02, shape) if lossy else 0.0)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_FUSED):
        e = iris.Engine(p, fw, precision=iris.FP32, stencil=st, dft_block=4)
        e.set_material(eps)
        if st == iris.STENCIL_FUSED:
            s = e.stepping()
            assert s["stencil"] == iris.STENCIL_FUSED and s["form"] == 1
            assert inside is None or (s["tile"], s["tiles"]) == inside
            assert slab is None or (s["slab_tile"], s["slab_tiles"]) == slab
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            e.set_field(which, q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape))
            for sl in (0, 1):
                v = e.pml_shape(sl)
                e.set_pml(which, sl, q.normal(size=v) + 1j * q.normal(size=v))
        e.step(150, 5)
        out.append([e.get_field(f)[1:-1, 1:-1, 1:-1] for f in (iris.E, iris.H)] +
                   [e.get_pml(f, sl) for f in (0, 1) for sl in (0, 1)] + [e.flux(0)])
        e.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (k, int(np.sum(a != b)))


@pytest.mark.parametrize("nx,ny", [(96, 42), (72, 57), (132, 30), (109, 21), (16, 29), (45, 11)])
def test_adjoint_shape_against_fp64(iris, tmp_path, nx, ny):
    """The adjoint's march on the same tiles: FP32 within rounding (1e-5 of the
    largest value over three steps) of the separate FP64 passes."""
    pml, planes = 5, 15
    nz, hi = planes + 2 * pml + 1, pml + 1
    w = cfg.Workload("adj", nx, ny, nz, pml, nz + 1 - pml, hi, 3, 2.25, 0, pml + 1, (1, nx, 1, ny, pml + 1, nz - pml), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.akx_re, p.aky_re, p.akz_re = 0.3, -0.7, 0.4
    r = np.random.default_rng(3)
    eps = 1.0 / r.uniform(1.0, 6.0, (p.hf - p.hi + 3, ny + 2, nx + 2))
    out = []
    for prec in (iris.FP64, iris.FP32):
        adj = iris.Adjoint(p, fw, (1, nx, 1, ny, hi, p.hf), precision=prec)
        adj.set_material(eps)
        A = adj.engine(1)
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            A.set_field(which, q.normal(size=A.field_shape) + 1j * q.normal(size=A.field_shape))
            for sl in (0, 1):
                v = A.pml_shape(sl)
                A.set_pml(which, sl, q.normal(size=v) + 1j * q.normal(size=v))
        adj.apply(3)
        out.append([A.get_field(f)[1:-1, 1:-1, 1:-1] for f in (iris.E, iris.H)] + [A.get_pml(f, s) for f in (0, 1) for s in (0, 1)])
        adj.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(a)), k
