"""The FP64 DFT block (integer digit products on the tensor cores): accumulators
against long-double sums of the sampled planes, at the edges of its tiles
(points, 32-frequency groups, 32-sample sub-blocks) and with rows whose
samples span many orders of magnitude or are zero.

Per number the block is off by at most half a unit of 2^-55 of the row's
largest sample (A and B digits: 2 x 2^-56 a term, two terms a sample) and the
final additions by 2^-53 of the sum; sin and cos differ by an ulp between
CUDA and glibc (2^-52 a term).  2^-50 dt sum_k max|F| holds all of them with
a margin of two."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("nx,ny,nof,block,steps", [(1, 1, 1, 0, 5), (7, 3, 33, 0, 32), (16, 8, 32, 40, 40),
                                                   (13, 11, 65, 100, 97), (23, 29, 20, 7, 45)])
def test_block_against_long_double(iris, tmp_path, nx, ny, nof, block, steps):
    w = cfg.Workload("d", nx, ny, 40, 4, 37, 18, 6, 2.25, 0, 9, (1, nx, 1, ny, 7, 33), nof, steps)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.dft_faces = iris.DFT_Z
    p.to_fourier = 170
    e = iris.Engine(p, fw, precision=iris.FP64, dft_block=block)
    r = np.random.default_rng(nof)
    shape = e.field_shape
    scale = 10.0 ** r.uniform(-12, 12, shape[1:3])  # neighbouring columns differ by many orders
    scale[ny // 2] = 0.0 if ny > 2 else scale[ny // 2]
    for which in (iris.E, iris.H):
        e.set_field(which, (r.normal(size=shape) + 1j * r.normal(size=shape)) * scale[None, :, :, None])
    planes, times = [], []
    for it in range(170, 170 + steps):
        e.step(it, 1)
        times.append(it + 1 - 170)
        planes.append([[e.get_plane(f, 3, z, (1, nx), (1, ny)) for z in (7, 33)] for f in (iris.E, iris.H)])
    got = e.get_fdata(0, 3)  # [iw, 12 * points]
    F = np.array(planes)     # [t, field, side, y, x, comp]
    F = F.transpose(0, 2, 3, 4, 1, 5).reshape(steps, 12 * nx * ny)  # side, location, component
    tw = np.exp(1j * (np.asarray(fw)[:, None] * np.asarray(times, dtype=np.float64)[None, :])).astype(np.complex128)
    want = (tw.astype(np.clongdouble) @ (F.astype(np.clongdouble) * np.longdouble(p.dt)))
    bound = 2.0 ** -50 * p.dt * np.abs(F).max(0) * steps
    err = np.abs((got - want).astype(np.complex128)).max(0)
    assert np.all(err <= bound), float(np.max(err / np.maximum(bound, 1e-300)))
    assert np.all(got[:, np.abs(F).max(0) == 0] == 0)
    e.close()
