"""Graph replay with the fused pass after an odd number of single steps: the two
buffer sets have exchanged their roles, and a block must not be replayed from
the graph that was captured on the other set.  Bit for bit the launches one by
one, in the single engine (the odd steps before the first sample, or a commit
in the middle of a block) and in a batch."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


def workload(iris, tmp_path, nx, ny, nz):
    w = cfg.Workload("g", nx, ny, nz, 5, nz - 4, 14, 6, 2.25, 0, 9, (1, nx, 1, ny, 7, nz - 7), 5, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.akx_re, p.precision, p.dft_faces, p.dft_block = 0.3, iris.FP32, iris.DFT_Z, 4
    return p, fw


@pytest.mark.parametrize("kernel", [0, 1])
def test_engine_blocks_on_both_sets(iris, tmp_path, kernel):
    p, fw = workload(iris, tmp_path, 37, 21, 64)
    out = []
    for graph in (False, True):
        e = iris.Engine(p, fw, precision=iris.FP32, stencil=iris.STENCIL_FUSED, dft_block=4, dft_kernel=kernel, graph=graph)
        e.material_pattern(3, 0.5)
        it = 150
        for n in (9, 8, 3, 13, 4, 1, 8):  # blocks start on one set, then on the other
            e.step(it, n)
            it += n
            e.dft_commit()
        out.append([e.get_field(f)[1:-1, 1:-1, 1:-1] for f in (iris.E, iris.H)] + [e.get_fdata(0, 3), e.flux(0)])
        e.close()
    assert np.any(out[0][0])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), k


def test_batch_blocks_on_both_sets(iris, tmp_path):
    sizes = [(37, 21, 64), (20, 33, 50)]
    ps = []
    for s in sizes:
        p, fw = workload(iris, tmp_path, *s)
        ps.append(p)
    out = []
    for graph in (False, True):
        b = iris.Batch(ps, fw, precision=iris.FP32, dft_faces=iris.DFT_Z, dft_block=4, graph=graph)
        for c in range(len(sizes)):
            b.material_pattern(c, 3 + c, 0.5)
        b.set_tile(7)
        it = 150
        for n in (9, 8, 3, 13, 4, 1, 8):
            b.step(it, n)
            it += n
            b.dft_commit()
        out.append([b.get_field(c, f)[1:-1, 1:-1, 1:-1] for c in range(len(sizes)) for f in (iris.E, iris.H)] +
                   [b.flux(c) for c in range(len(sizes))])
        b.close()
    assert np.any(out[0][0])
    for k, (x, y) in enumerate(zip(*out)):
        assert np.array_equal(x, y), k
