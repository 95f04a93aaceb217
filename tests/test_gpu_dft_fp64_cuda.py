"""The FP64 DFT block on the CUDA cores (IRIS_DFT_KERNEL_CUDA): one sample after
another into the accumulators, so block lengths and flux reads in between leave
no trace; against long-double sums of the sampled planes.

A real number takes two FMAs a sample, each off by 2^-53 of a partial sum of at
most 2 n dt max|F| over n samples: n 2^-51 n dt max|F|, times sqrt(2) for the
complex one; dt F and the twiddle bring 2^-53 and 2^-52 a term.  n^2 2^-50 dt
max|F| holds them for n = 37."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("nx,ny,nof", [(1, 1, 1), (7, 3, 9), (13, 11, 33)])
def test_sums_do_not_depend_on_blocks(iris, tmp_path, nx, ny, nof, steps=37):
    w = cfg.Workload("d", nx, ny, 40, 4, 37, 18, 6, 2.25, 0, 9, (1, nx, 1, ny, 7, 33), nof, steps)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.dft_faces, p.to_fourier = iris.DFT_Z, 170
    out = []
    for block, reads in ((1, 0), (7, 0), (32, 5), (256, 11)):
        e = iris.Engine(p, fw, precision=iris.FP64, dft_block=block, dft_kernel=iris.DFT_KERNEL_CUDA)
        r = np.random.default_rng(nof)
        for which in (iris.E, iris.H):
            e.set_field(which, r.normal(size=e.field_shape) + 1j * r.normal(size=e.field_shape))
        planes, times = [], []
        for it in range(170, 170 + steps):
            e.step(it, 1)
            if reads and it % reads == 0:
                e.flux(0)
                assert e.info()["dft_buffered"] == 0
            times.append(it + 1 - 170)
            planes.append([[e.get_plane(f, 3, z, (1, nx), (1, ny)) for z in (7, 33)] for f in (iris.E, iris.H)])
        out.append((e.get_fdata(0, 3), e.flux(0)))
        e.close()
    for a, J in out[1:]:
        assert np.array_equal(a, out[0][0]) and np.array_equal(J, out[0][1])
    F = np.array(planes).transpose(0, 2, 3, 4, 1, 5).reshape(steps, 12 * nx * ny)
    tw = np.exp(1j * (np.asarray(fw)[:, None] * np.asarray(times, dtype=np.float64)[None, :])).astype(np.complex128)
    want = tw.astype(np.clongdouble) @ (F.astype(np.clongdouble) * np.longdouble(p.dt))
    err = np.abs((out[0][0] - want).astype(np.complex128)).max(0)
    assert np.all(err <= 2.0 ** -50 * p.dt * np.abs(F).max(0) * steps ** 2)
