"""Spans of one step on grids that step in the resident kernel by default: the
split passes take them, and any mix of call lengths gives the same bits as
either stepping alone (calls of one step, a ring that fills after one, a last
step left over by a block)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny,nz,ipol,lossy", [(1, 1, 60, 2, False), (4, 4, 128, 2, False), (61, 11, 36, 2, True), (40, 1, 64, 1, False)])
@pytest.mark.parametrize("block,calls", [(8, (1, 1, 1, 9, 1, 5, 1)), (1, (3, 1, 2)), (4, (5, 5, 1))])
def test_mixed_spans_equal_split(iris, tmp_path, precision, nx, ny, nz, ipol, lossy, block, calls):
    pml = 5
    w = cfg.Workload("one", nx, ny, nz, pml, nz + 1 - pml, nz // 2 - 3, 6, 2.25, 0, pml + 4,
                     (1, nx, 1, ny, pml + 1, nz - pml), 5, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, i_pol=ipol))
    p.akx_re = 0.3
    r = np.random.default_rng(3)
    shape = (p.hf - p.hi + 3, ny + 2, nx + 2)
    eps = 1.0 / r.uniform(1.0, 6.0, shape) + (1j * r.uniform(-0.02, 0.02, shape) if lossy else 0.0)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_PERSISTENT, iris.STENCIL_DEFAULT):
        e = iris.Engine(p, fw, precision=precision, stencil=st, dft_block=block)
        e.set_material(eps)
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            e.set_field(which, q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape))
        e.timing_start()
        it = 150
        for n in calls:
            e.step(it, n)
            it += n
        k = e.timing_read()[2]
        if st == iris.STENCIL_DEFAULT:
            # spans end where the ring of `block` samples fills
            spans, left = [], block
            for n in calls:
                while n:
                    m = min(n, left)
                    spans.append(m)
                    n -= m
                    left = left - m or block
            ones = sum(m == 1 for m in spans)
            assert (k["update_e"], k["persistent"]) == (ones, len(spans) - ones)
        out.append([e.get_field(f) for f in (iris.E, iris.H)] + [e.get_pml(f, s) for f in (0, 1) for s in (0, 1)] +
                   [e.get_fdata(0, 3), e.flux(0)])
        e.close()
    for other in out[1:]:
        for k, (a, b) in enumerate(zip(out[0], other)):
            assert np.array_equal(a, b), (k, int(np.sum(a != b)))
