"""The FP64 default steps with the persistent kernels where the estimates say
they are the faster, with the split passes elsewhere, and gives the same
state bit for bit whichever it takes: a grid of few long rows (a row a CTA), one
just too large for shared memory, small ones."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("nx,ny,nz,kind", [(16, 4, 64, "persistent"), (2600, 1, 16, "persistent"),
                                           (2600, 1, 64, "update_e"), (70, 70, 70, "persistent"),
                                           (20, 20, 1000, "update_e"), (257, 40, 103, "update_e")])
def test_fp64_default(iris, tmp_path, nx, ny, nz, kind):
    w = cfg.Workload("choice", nx, ny, nz, 4, nz - 3, nz // 2, 2, 2.25, 0, 6, (1, nx, 1, ny, 5, nz - 4), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=2))
    p.akx_re, p.dft_faces = 0.3, iris.DFT_Z
    out = []
    for st in (iris.STENCIL_DEFAULT, iris.STENCIL_PERSISTENT, iris.STENCIL_SPLIT):
        e = iris.Engine(p, fw, precision=iris.FP64, stencil=st, dft_block=4)
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            e.set_field(which, q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape))
        e.timing_start()
        e.step(150, 3)
        n = e.timing_read()[2]
        if st == iris.STENCIL_DEFAULT:
            assert n[kind] > 0 and sum(n[k] > 0 for k in ("persistent", "update_e")) == 1
        out.append([e.get_field(f) for f in (iris.E, iris.H)] + [e.flux(0)])
        e.close()
    for a in out[1:]:
        for u, v in zip(out[0], a):
            assert np.array_equal(u, v)
