"""Flux reads with one to a full ring of FP64 samples pending: up to three are
accumulated one after another, more are added on the fly and stay; the flux is
that of an engine with its samples committed step by step and read once, within
rounding, and so are the accumulators.

Both sum the same samples: per number n samples, each path off by at most
n 2^-50 dt max|F| (the FMA path n / 2 times that, n <= 40), so J, a sum of
products of two accumulators over the face, is relative to sum |a||b| + |c||d|
off by 4 n^2 2^-51."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("nx,ny,nof,calls", [(4, 4, 33, (1,) * 40), (13, 9, 20, (3, 1, 4, 2, 5, 8, 3, 7, 1, 1, 5)), (1, 1, 200, (2,) * 20)])
def test_flux_after_every_call(iris, tmp_path, nx, ny, nof, calls):
    w = cfg.Workload("d", nx, ny, 60, 4, 57, 25, 8, 2.25, 0, 9, (1, nx, 1, ny, 7, 53), nof, 40)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.dft_faces, p.to_fourier = iris.DFT_Z, 170
    n = sum(calls)
    engines = [iris.Engine(p, fw, precision=iris.FP64, dft_block=b, dft_kernel=k)
               for b, k in ((0, iris.DFT_KERNEL_AUTO), (1, iris.DFT_KERNEL_AUTO), (32, iris.DFT_KERNEL_CUDA))]
    r = np.random.default_rng(3)
    for which in (iris.E, iris.H):
        f = r.normal(size=engines[0].field_shape) + 1j * r.normal(size=engines[0].field_shape)
        for e in engines:
            e.set_field(which, f)
    it, pending, e = 170, 0, engines[0]
    for c in calls:
        for x in engines:
            x.step(it, c)
        it += c
        pending = (pending + c) % 32 if pending + c >= 32 else pending + c
        assert e.info()["dft_buffered"] == pending
        J = e.flux(0)
        if pending <= 3:
            pending = 0
        assert e.info()["dft_buffered"] == pending
    want = engines[2].flux(0)  # one sample after another
    F = [x.get_fdata(0, 3) for x in engines]
    assert np.array_equal(F[1], F[2])  # blocks of one are the same
    m = np.abs(F[2]).max()
    assert np.abs(F[0] - F[2]).max() <= 4 * n * n * 2.0 ** -51 * m * np.sqrt(n)
    for side in (4, 5):
        a = F[2].reshape(nof, 2, nx * ny, 6)[:, side - 4]
        size = p.eps0 * p.Q / (2 * p.dt) * (np.abs(a[..., 0] * a[..., 4]) + np.abs(a[..., 1] * a[..., 3])).sum(1)
        assert np.all(np.abs(J[side] - want[side]) <= 4 * n * n * 2.0 ** -51 * np.sqrt(n) * size.max())
    for x in engines:
        x.close()


@pytest.mark.parametrize("block", [1, 3])
def test_short_blocks_replayed_from_a_graph(iris, tmp_path, block):
    w = cfg.Workload("d", 13, 9, 60, 4, 57, 25, 8, 2.25, 0, 9, (1, 13, 1, 9, 7, 53), 20, 40)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    out = []
    for graph in (False, True):
        e = iris.Engine(p, fw, precision=iris.FP64, stencil=iris.STENCIL_SPLIT, dft_block=block, graph=graph)
        e.step(150, 3 * block)  # the first commit is recorded, the others replay it
        e.step(150 + 3 * block, 2)
        out.append([e.get_fdata(0, j) for j in (1, 2, 3)] + [e.flux(0), e.get_field(iris.E)])
        e.close()
    assert np.any(out[0][0])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
