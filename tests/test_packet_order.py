"""The order of the resident kernel's packet exchange: one place a number holds
the packets of all steps, so no lane may still wait for a packet when it is
overwritten.  The model is a border between two CTAs: an E pair on one side, the
H pair it exchanges with on the other, every interleaving of their single reads
and publications explored.  A lane reads the parts that ``reads`` names; where
a material mixes the parts, the pair exchanges them before either publishes."""
import importlib

import numpy as np
import pytest

cfg = importlib.import_module("irisfdtd-academic_gb300.configs")


def stuck(reads_e, reads_h, pair_e, steps=3):
    """Whether some interleaving leaves a lane waiting for a tag that has passed.
    Lane (side, p) a step: read reads[p] (E of step s waits for H's tag s - 1,
    H for E's tag s), meet its partner if pair, publish its part with tag s."""
    progs = {}
    for side, reads in (("E", reads_e), ("H", reads_h)):
        for p in (0, 1):
            ops = []
            for s in range(1, steps + 1):
                want = s - 1 if side == "E" else s
                if want > 0:  # the first E phase reads the state in memory
                    ops += [("read", ("H" if side == "E" else "E", q), want) for q in reads(p)]
                if side == "E" and pair_e:
                    ops.append(("meet",))
                ops.append(("publish", (side, p), s))
            progs[side, p] = ops
    lanes = sorted(progs)
    start = (tuple(0 for _ in lanes), tuple(0 for _ in lanes))  # program counters, tags by (side, part)
    seen, todo = {start}, [start]
    while todo:
        pc, tag = todo.pop()
        for k, lane in enumerate(lanes):
            if pc[k] == len(progs[lane]):
                continue
            op = progs[lane][pc[k]]
            moved, t = [k], tag
            if op[0] == "read":
                have = tag[lanes.index(op[1])]
                if have > op[2]:
                    return True
                if have < op[2]:
                    continue
            elif op[0] == "meet":
                other = lanes.index((lane[0], 1 - lane[1]))
                if pc[other] != pc[k]:
                    continue
                moved = [k, other]
            else:
                t = tag[:k] + (op[2],) + tag[k + 1:]
            new = (tuple(c + (i in moved) for i, c in enumerate(pc)), t)
            if new not in seen:
                seen.add(new)
                todo.append(new)
    return not any(all(pc[k] == len(progs[lane]) for k, lane in enumerate(lanes)) for pc, _ in seen)


def own(p):
    return [p]


def both(p):
    return [0, 1]


def test_packet_order():
    assert not stuck(own, own, False)  # real material
    assert not stuck(own, own, True)   # complex material: the other part from the pair
    assert not stuck(both, both, False) and not stuck(both, both, True)  # images with a phase
    # an E lane that reads a part its publication does not answer for may wait
    # for a packet that has been overwritten
    assert stuck(both, own, False)


# nx, ny, nz, pml, ak, steps: rows alone on their CTA, y rows of one plane on several
# CTAs, a phase across z only, across y only, one step a launch
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,pml,ak,steps", [(3, 1, 120, 4, (0, 0, 0), 60), (5, 7, 40, 3, (0.3, 0, 0), 40),
                                                   (2, 60, 20, 4, (0, 0, 0), 30), (2, 60, 20, 4, (0, 0.5, 0), 30),
                                                   (4, 4, 64, 3, (0, 0, 0.4), 1), (7, 33, 16, 3, (0, 0, 0), 1)])
def test_complex_material_packets_equal_split(iris, tmp_path, nx, ny, nz, pml, ak, steps):
    w = cfg.Workload("lossy", nx, ny, nz, pml, nz + 1 - pml, pml + 1, nz - 2 * pml - 1, 2.25, 0, pml + 2,
                     (1, nx, 1, ny, pml + 1, nz - pml), 5, steps)
    p, fw, _ = iris.setparam(cfg.write_input(str(tmp_path / "in.dat"), w))
    p.akx_re, p.aky_re, p.akz_re = ak
    r = np.random.default_rng(3)
    shape = (p.hf - p.hi + 3, ny + 2, nx + 2)
    eps = 1.0 / r.uniform(1.0, 6.0, shape) + 1j * r.uniform(-0.02, 0.02, shape)
    out = []
    for st in (iris.STENCIL_SPLIT, iris.STENCIL_PERSISTENT):
        e = iris.Engine(p, fw, precision=iris.FP64, stencil=st)
        e.set_material(eps)
        q = np.random.default_rng(4)
        for which in (iris.E, iris.H):
            e.set_field(which, q.normal(size=e.field_shape) + 1j * q.normal(size=e.field_shape))
        e.step(150, steps)
        e.step(150 + steps, 1)
        out.append([e.get_field(f) for f in (iris.E, iris.H)] + [e.get_pml(f, s) for f in (0, 1) for s in (0, 1)])
        e.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), (k, int(np.sum(a != b)))
