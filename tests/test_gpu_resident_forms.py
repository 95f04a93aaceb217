"""The forms of the resident kernel: the cases of the tests that ask for it run it
(not the kernel with grid-wide barriers, which gives the same bits), with
packets where they are about packets; and the forms that only large or
slab-heavy grids take (E_x, or D and B, left in global memory, in both
precisions, with and without runs of 32 cells a warp) equal the split passes."""
import importlib

import numpy as np
import pytest

import test_gpu_resident as resident
import test_gpu_resident_packets as packets

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


def engine(iris, tmp_path, case, precision, stencil):
    nx, ny, nz, pml, zi, pol, ak, lossy, n = case
    w = cfg.Workload("form", nx, ny, nz, pml, nz + 1 - pml, nz // 2 - 3, 6, 2.25, 0, zi,
                     (1, nx, 1, ny, pml + 1, nz - pml), 5, n)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=pol))
    (p.akx_re, p.akx_im), (p.aky_re, p.aky_im), (p.akz_re, p.akz_im) = [(complex(a).real, complex(a).imag) for a in ak]
    return iris.Engine(p, fw, precision=precision, stencil=stencil, dft_block=4)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", resident.CASES)
def test_cases_run_the_resident_kernel(iris, tmp_path, name, precision):
    e = engine(iris, tmp_path, resident.CASES[name], precision, iris.STENCIL_PERSISTENT)
    s = e.stepping()
    # (in FP64 770 thousand cells do not fit; FORMS has a smaller one)
    fits = not (name == "ex_in_global_memory" and precision == iris.FP64)
    assert s["stencil"] == iris.STENCIL_PERSISTENT and (s["form"] > 0) == fits
    if name == "ex_in_global_memory" and fits:
        assert s["components"] == 5
    e.close()


@pytest.mark.parametrize("name", packets.CASES)
def test_cases_exchange_packets(iris, tmp_path, name):
    e = engine(iris, tmp_path, packets.CASES[name], iris.FP64, iris.STENCIL_PERSISTENT)
    assert e.stepping()["form"] == 2
    e.close()


# precision, case, components in shared memory, D and B there, runs
FORMS = {
    "fp64_ex_global": (0, (250, 4, 340, 16, 40, 2, (0.1, 0, 0), False, 5), 5, True, False),
    "fp64_ex_global_lossy": (0, (250, 4, 340, 16, 40, 1, (0.1, 0, 0.2), True, 5), 5, True, False),
    "fp64_slabs_global": (0, (100, 10, 207, 97, 101, 2, (0.3, 0.2, 0), False, 5), 6, False, False),
    "fp32_ex_global_no_runs": (1, (40, 10, 1850, 30, 50, 2, (0.1, 0, 0), True, 5), 5, True, False),
    "fp32_slabs_and_ex_global_no_runs": (1, (40, 10, 2000, 30, 50, 2, (0.1, 0, 0), True, 5), 5, False, False),
    "fp32_slabs_global": (1, (100, 10, 420, 200, 204, 2, (0.3, 0.2, 0), False, 5), 6, False, True),
    "fp32_slabs_global_no_runs": (1, (40, 10, 1050, 500, 504, 2, (0.3, 0.2, 0), False, 5), 6, False, False),
    "fp32_slabs_and_ex_global": (1, (100, 10, 760, 370, 374, 2, (0.3, 0, 0.1), False, 5), 5, False, True),
}


@pytest.mark.parametrize("name", FORMS)
def test_form_equals_split(iris, tmp_path, name):
    precision, case, components, upml, runs = FORMS[name]
    nx, ny, nz, lossy, n = case[0], case[1], case[2], case[7], case[8]
    r = np.random.default_rng(3)
    eps = 1.0 / r.uniform(1.0, 6.0, (8, ny + 2, nx + 2)) + (1j * r.uniform(-0.02, 0.02, (8, ny + 2, nx + 2)) if lossy else 0.0)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_PERSISTENT):
        e = engine(iris, tmp_path, case, precision, st)
        e.set_material(eps)
        if st == iris.STENCIL_PERSISTENT:
            s = e.stepping()
            assert s["form"] == 1 and (s["components"], s["upml_resident"], s["runs"]) == (components, upml, runs), s
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            e.set_field(which, q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape))
            for slab in (0, 1):
                v = e.pml_shape(slab)
                e.set_pml(which, slab, q.normal(size=v) + 1j * q.normal(size=v))
        e.step(150, 1)
        e.step(151, n)
        out.append([e.get_field(f) for f in (iris.E, iris.H)] + [e.get_pml(f, s) for f in (0, 1) for s in (0, 1)] +
                   [e.flux(0)] + [e.get_fdata(0, j) for j in (1, 2, 3)])
        e.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (k, int(np.sum(a != b)))
