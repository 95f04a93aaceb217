"""The engine that holds the adjoint state (iris_adjoint_engine, which = 1) may
be stepped like any other: bit for bit a split-pass engine from the same state,
source included, also after the adjoint recursion has swapped its buffers.  It
takes no DFT samples and says so."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("swaps", [0, 1])
def test_adjoint_engine_steps_with_its_source(iris, tmp_path, precision, swaps):
    nx, ny, nz = 12, 10, 48
    w = cfg.Workload("adj", nx, ny, nz, 5, 44, 20, 4, 2.25, 0, 9, (1, nx, 1, ny, 7, 42), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.akx_re = 0.3
    adj = iris.Adjoint(p, fw, (2, 9, 2, 8, 20, 23), precision=precision)
    A = adj.engine(1)
    e = iris.Engine(p, fw, precision=precision, stencil=iris.STENCIL_SPLIT)
    adj.apply(swaps)
    q = np.random.default_rng(4)
    for which in (iris.E, iris.H):
        f = q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape)
        A.set_field(which, f)
        e.set_field(which, f)
        for slab in (0, 1):
            v = q.normal(size=e.pml_shape(slab)) + 1j * q.normal(size=e.pml_shape(slab))
            A.set_pml(which, slab, v)
            e.set_pml(which, slab, v)
    for x in (A, e):
        x.step(160, 5)
        x.tfsf(165)
        x.step(166, 1)
        x.sync()
    for which in (iris.E, iris.H):
        assert np.array_equal(A.get_field(which), e.get_field(which)), which
    for call in (lambda: A.flux(0), lambda: A.get_fdata(0, 3)):
        with pytest.raises(iris.IrisError) as x:
            call()
        assert x.value.code == -1
    adj.close()
    e.close()
