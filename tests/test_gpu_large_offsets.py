"""FP32 grids whose three components lie past 32-bit offsets (more than 2^31
elements): the fused pass steps them with one column of registers a thread
instead of the staged tiles, in the single engine and in a batch.  A cell of
1021x1019x700 (its last tiles ragged on both axes) against the split passes, bit
for bit, on planes of every axis, in the structure, both slabs and behind them,
and its fluxes; the batch takes it beside a small cell that is staged.  36 GB of
fields for the split passes, 72 GB for the fused pass."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")

NX, NY, NZ, PML, STEPS = 1021, 1019, 700, 8, 36


def params(iris, tmp_path, nx, ny, nz):
    w = cfg.Workload("large", nx, ny, nz, PML, nz + 1 - PML, 16, 20, 2.25, 0, PML + 3, (1, nx, 1, ny, PML + 2, 40), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.akx_re, p.aky_re, p.akz_re, p.dft_faces = 0.3, -0.7, 0.4, iris.DFT_Z
    p.dft_block = 8
    return p, fw


def run(iris, p, fw, stencil, eps):
    e = iris.Engine(p, fw, precision=iris.FP32, stencil=stencil, dft_block=8)
    assert 3 * e.info()["comp_elems"] >= 2 ** 31
    if eps is None:
        e.material_pattern(5, 0.5)
    else:
        e.set_material(eps)
    e.timing_start()
    e.step(150, STEPS)
    k = e.timing_read()[2]
    out = {}
    for which in (iris.E, iris.H):
        for z in (0, 1, PML - 1, PML + 1, 17, 35, 43, NZ - 3, NZ):
            out[which, 3, z] = e.get_plane(which, 3, z, (1, NX), (1, NY))
        out[which, 2, 512] = e.get_plane(which, 2, 512, (0, NX), (1, NZ))
        out[which, 1, 1] = e.get_plane(which, 1, 1, (0, NY), (1, NZ))
        out[which, 1, NX] = e.get_plane(which, 1, NX, (0, NY), (1, NZ))
    out["flux"] = e.flux(0)
    e.close()
    return out, k


@pytest.mark.parametrize("lossy", [False, True])
def test_large_cell_fused_equals_split(iris, tmp_path, lossy):
    p, fw = params(iris, tmp_path, NX, NY, NZ)
    eps = None
    if lossy:
        r = np.random.default_rng(3)
        shape = (p.hf - p.hi + 3, NY + 2, NX + 2)
        eps = np.empty(shape, dtype=complex)
        eps.real, eps.imag = r.uniform(0.2, 1.0, shape), r.uniform(-0.02, 0.02, shape)
    want, k = run(iris, p, fw, iris.STENCIL_SPLIT, eps)
    assert k["update_e"] == STEPS
    got, k = run(iris, p, fw, iris.STENCIL_DEFAULT, eps)
    assert k["fused_eh"] == STEPS and k["update_e"] == 0
    for key in want:
        assert np.array_equal(want[key], got[key]), key
    for which in (iris.E, iris.H):
        assert all(np.any(want[which, 3, z]) for z in (1, PML - 1, 17, 35, NZ - 3))
        # the structure makes the planes vary across the tiles
        assert np.std(np.abs(want[which, 3, 17][..., 0])) > 0 or np.std(np.abs(want[which, 3, 17][..., 1])) > 0
    assert np.any(want["flux"][4]) and np.any(want["flux"][5])


def test_large_cell_in_a_batch(iris, tmp_path):
    cells = [(NX, NY, NZ), (45, 37, 90)]
    ps, want = [], []
    for c in cells:
        p, fw = params(iris, tmp_path, *c)
        p.precision = iris.FP32
        ps.append(p)
        e = iris.Engine(p, fw, precision=iris.FP32, stencil=iris.STENCIL_SPLIT, dft_block=8)
        e.material_pattern(7, 0.4)
        e.step(150, STEPS)
        want.append(e.flux(0))
        e.close()
    b = iris.Batch(ps, fw, precision=iris.FP32, dft_faces=iris.DFT_Z, dft_block=8)
    for c in range(len(cells)):
        b.material_pattern(c, 7, 0.4)
    b.set_tile(7)
    b.step(150, STEPS)
    for c in range(len(cells)):
        assert np.any(want[c][5]) and np.array_equal(b.flux(c), want[c]), c
    b.close()
