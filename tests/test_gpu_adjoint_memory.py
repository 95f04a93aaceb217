"""The gradient where its checkpoints need the memory of the marched step's second
field buffers: they are given back in the middle of the forward solve and the
backward one steps in place, with the same gradient but for FP32 rounding (a
step's separate passes against the march: 1e-5 of the largest value); where even
that is not enough the call returns IRIS_ENOMEM and a smaller one still runs.
Device memory is filled by a tensor that leaves room for three and a half
checkpoints."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


def test_checkpoints_take_the_second_buffers(iris, tmp_path):
    torch = pytest.importorskip("torch")
    nx, ny, nz, pml, every, steps = 220, 210, 260, 6, 40, 160
    w = cfg.Workload("mem", nx, ny, nz, pml, nz + 1 - pml, 16, 4, 2.25, 0, 10, (1, nx, 1, ny, 8, 24), 3, 9)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w, pulse_steps=20.0))
    p.akx_re = 0.3
    design = (5, 200, 7, 190, 16, 19)
    eta = 1.0 / np.random.default_rng(3).uniform(1.0, 6.0, (4, 184, 196))

    def gradient(adj, n):
        adj.set_design(eta)
        L, _ = adj.forward(n)
        return L, adj.backward()

    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    adj = iris.Adjoint(p, fw, design, checkpoint_every=every, precision=iris.FP32)
    L0, g0 = gradient(adj, steps)
    assert np.max(np.abs(g0)) > 0
    adj.close()
    adj = iris.Adjoint(p, fw, design, checkpoint_every=every, precision=iris.FP32)
    fields = 2 * 3 * adj.engine(0).info()["comp_elems"] * 8
    one = fields + 2 * 3 * nx * ny * (pml + pml) * 8  # a checkpoint: E, H, D, B
    gradient(adj, 1)
    before = free()  # one checkpoint is there
    fill = torch.empty(before - int(2.5 * one), dtype=torch.uint8, device="cuda")
    left = free()
    L1, g1 = gradient(adj, steps)
    # three more checkpoints and both second buffers back
    assert abs((left - free()) - (3 * one - fields)) < 0.1 * one
    assert L1 == L0
    assert np.max(np.abs(g1 - g0)) <= 1e-5 * np.max(np.abs(g0))
    with pytest.raises(iris.IrisError) as x:
        adj.forward(2 * steps)
    assert x.value.code == -2
    L2, g2 = gradient(adj, steps)
    assert L2 == L0 and np.array_equal(g2, g1)
    del fill
    torch.cuda.empty_cache()
    adj.close()
