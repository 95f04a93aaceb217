"""The FP64 DFT block where its sums leave the normal range: fields so small that
samples and sums are subnormal, and so large that the sums end just below the
largest double; against long-double sums of the sampled planes.

As in the normal range a number is off by at most 2^-50 dt sum_k max|F|; a
block's sum and each of the additions add half of 2^-1074."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("lo,hi,block,steps", [(-322, -300, 0, 45), (-312, -304, 7, 20), (-309, -305, 40, 33), (308.2, 308.2, 0, 3)])
def test_block_at_the_ends_of_the_range(iris, tmp_path, lo, hi, block, steps, nx=7, ny=5, nof=20):
    w = cfg.Workload("d", nx, ny, 40, 4, 37, 18, 6, 2.25, 0, 9, (1, nx, 1, ny, 7, 33), nof, steps)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, epump=0.0))
    p.dft_faces, p.to_fourier = iris.DFT_Z, 170
    e = iris.Engine(p, fw, precision=iris.FP64, dft_block=block)
    r = np.random.default_rng(nof)
    shape = e.field_shape
    if lo > 0:  # uniform: nothing moves at the planes within the steps
        f = np.full(shape, 10.0 ** lo)
    else:
        f = (r.normal(size=shape) + 1j * r.normal(size=shape)) * (10.0 ** r.uniform(lo, hi, shape[1:3]))[None, :, :, None]
    for which in (iris.E, iris.H):
        e.set_field(which, f)
    planes, times = [], []
    for it in range(170, 170 + steps):
        e.step(it, 1)
        times.append(it + 1 - 170)
        planes.append([[e.get_plane(g, 3, z, (1, nx), (1, ny)) for z in (7, 33)] for g in (iris.E, iris.H)])
    got = e.get_fdata(0, 3)
    F = np.array(planes).transpose(0, 2, 3, 4, 1, 5).reshape(steps, 12 * nx * ny)
    tw = np.exp(1j * (np.asarray(fw)[:, None] * np.asarray(times, dtype=np.float64)[None, :])).astype(np.complex128)
    want = tw.astype(np.clongdouble) @ (F.astype(np.clongdouble) * np.longdouble(p.dt))
    assert np.all(np.isfinite(got)) and np.any(got) and (lo < 0 or np.abs(got.real).max() > 2.0 ** 1023)
    m = np.abs(F.real).max(0) + np.abs(F.imag).max(0)
    bound = np.longdouble(2.0 ** -50) * np.longdouble(p.dt) * m * steps + np.longdouble(2) * steps * np.longdouble(5e-324)
    for a, b in ((got.real, want.real), (got.imag, want.imag)):
        assert np.all(np.abs(a.astype(np.longdouble) - b).max(0) <= bound)
    e.close()
