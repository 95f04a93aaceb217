"""The resident persistent kernel (grids whose E and H fit in the SMs' shared
memory): bit for bit the split passes from random states, ghosts included, at
the sizes where its partition can go wrong (fewer rows than SMs, fewer rows a
CTA than y rows, a last 32-cell run of one lane, E_x left in global memory),
with Bloch phases on every axis, both TF/SF variants and polarisations, a
source next to the UPML and no source."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")

# nx, ny, nz, pml, tfsf_zi, i_pol, ak, complex material, steps
CASES = {
    "column": (1, 1, 40, 4, 9, 2, (0, 0, 0), False, 9),
    "fewer_rows_than_sms": (3, 5, 28, 4, 8, 2, (0.3, 0, 0), False, 8),
    "rows_below_ny": (5, 190, 18, 3, 6, 2, (0.2 + 0.05j, 0, 0), False, 6),
    "one_lane_run": (33, 9, 48, 5, 12, 2, (0.3, -0.7, 0.4), False, 7),
    "narrow_rows_lossy": (13, 17, 40, 5, 11, 1, (0.5, 0, 0), True, 7),
    "lossy_runs": (61, 11, 36, 4, 10, 2, (0.5, 0.2, 0), True, 7),
    "variant2": (40, 1, 64, 6, 14, 2, (-0.4, 0, 0), False, 7),
    "variant1_row": (40, 1, 64, 6, 14, 1, (0, 0, 0), False, 7),
    "source_at_2": (24, 6, 30, 3, 2, 2, (0, 0, 0), False, 6),
    "no_source": (24, 6, 30, 3, 8, 3, (0.1, 0.2, 0), False, 6),
    "ex_in_global_memory": (250, 4, 770, 16, 40, 2, (0.1, 0, 0), False, 5),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", CASES)
def test_resident_equals_split(iris, tmp_path, name, precision):
    nx, ny, nz, pml, zi, pol, ak, lossy, n = CASES[name]
    hi, dh = nz // 2 - 3, 6
    w = cfg.Workload(name, nx, ny, nz, pml, nz + 1 - pml, hi, dh, 2.25, 0, zi, (1, nx, 1, ny, pml + 1, nz - pml), 5, n)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=pol))
    (p.akx_re, p.akx_im), (p.aky_re, p.aky_im), (p.akz_re, p.akz_im) = [(complex(a).real, complex(a).imag) for a in ak]
    r = np.random.default_rng(3)
    eps = 1.0 / r.uniform(1.0, 6.0, (dh + 2, ny + 2, nx + 2)) + (1j * r.uniform(-0.02, 0.02, (dh + 2, ny + 2, nx + 2))
                                                                 if lossy else 0.0)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_PERSISTENT):
        e = iris.Engine(p, fw, precision=precision, stencil=st, dft_block=4)
        e.set_material(eps)
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            e.set_field(which, q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape))
            for slab in (0, 1):
                shape = e.pml_shape(slab)
                e.set_pml(which, slab, q.normal(size=shape) + 1j * q.normal(size=shape))
        e.step(150, 1)  # every neighbour of the first step is a stored ghost
        e.step(151, n)
        out.append([e.get_field(f) for f in (iris.E, iris.H)] +
                   [e.get_pml(f, s) for f in (0, 1) for s in (0, 1)] + [e.flux(0)] +
                   [e.get_fdata(0, j) for j in (1, 2, 3)])
        e.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (k, int(np.sum(a != b)))
