"""The FP32 adjoint step with its interior planes marched against the FP64 one
(separate passes, in place), from random states with Bloch phases on every
axis: tiles with and without borders, one cell and one row of cells past a
tile, chunk ends, and too few planes to march.  A step adds and scales a few
values of magnitude 1 with factors below 1: FP32 rounding stays within 1e-5 of
the largest value over three steps."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("nx,ny,planes", [(12, 10, 14), (33, 15, 15), (54, 8, 41), (55, 9, 3), (163, 25, 29), (97, 44, 13),
                                          (1, 40, 28), (40, 1, 14), (17, 30, 2)])
def test_adjoint_march_against_fp64(iris, tmp_path, nx, ny, planes):
    pml = 5
    nz = planes + 2 * pml + 1  # planes pml + 2 .. nz - 1 - pml march: planes - 1
    hi = pml + 1
    w = cfg.Workload("adj", nx, ny, nz, pml, nz + 1 - pml, hi, 1, 2.25, 0, pml + 1, (1, nx, 1, ny, pml + 1, nz - pml), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.akx_re, p.aky_re, p.akz_re = 0.3, -0.7, 0.4
    r = np.random.default_rng(3)
    eps = 1.0 / r.uniform(1.0, 6.0, (p.hf - p.hi + 3, ny + 2, nx + 2))
    inner = (slice(1, nz + 1), slice(1, ny + 1), slice(1, nx + 1))
    out = []
    for prec in (iris.FP64, iris.FP32):
        adj = iris.Adjoint(p, fw, (1, nx, 1, ny, hi, p.hf), precision=prec)
        adj.set_material(eps)
        A = adj.engine(1)
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            A.set_field(which, q.normal(size=A.field_shape) + 1j * q.normal(size=A.field_shape))
            for slab in (0, 1):
                s = A.pml_shape(slab)
                A.set_pml(which, slab, q.normal(size=s) + 1j * q.normal(size=s))
        adj.apply(3)
        out.append([A.get_field(f)[inner] for f in (iris.E, iris.H)] + [A.get_pml(f, s) for f in (0, 1) for s in (0, 1)])
        adj.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(a)), k
