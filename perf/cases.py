"""What a user of this framework has it do, as measurable cases.

A case is a dict of plain values; ``prepare`` builds what a user's program
holds before the call (an engine, a batch, a gradient object or a run
directory, with its inputs drawn from a seed), ``run`` makes one pass through
the public entry points, ``work`` counts what the pass cannot do without and
``exact`` computes the same outputs in 64 bits with plain torch operations.

FP32-mode outputs are returned in FP32, the precision they are computed in.
"""
from __future__ import annotations

import importlib
import math
import os
import shutil
import tempfile

import numpy as np
import torch

os.environ.setdefault("IRIS_QUIET", "1")  # iris_run_input's progress lines
iris = importlib.import_module("irisfdtd-academic_gb300")
cfg = importlib.import_module("irisfdtd-academic_gb300.configs")

# the chip's own memory (registers and shared memory): a state smaller than
# this has to be read and written once a pass, a larger one once a step
ON_CHIP_BYTES = 64e6


def listed():
    return [
        # the drop-in program on the reference's film example: a 1x1x400 column read from inputFDTD.dat,
        # 500 wavelengths, FP64, spectra files written (example_1's deck with fewer steps)
        dict(name="deck_film_1x1x400_fp64", kind="deck", nx=1, ny=1, nz=400, pml=75, nof=500, steps=1500, outputs=3),
        # the smallest 3D cell, launch- and latency-bound: 4x4x512 FP64 slab, R and T planes at 200 frequencies
        dict(name="slab_4x4x512_fp64", kind="engine", prec=64, nx=4, ny=4, nz=512, faces="z", nof=200, steps=256,
             block=32, structure="slab", ipol=2, kx=0.0, fields=1, plane=0),
        # the slit array of example_2's form, FP32: one period of a grating, R and T planes at 300 frequencies
        dict(name="slit_256x4x768_fp32", kind="engine", prec=32, nx=256, ny=4, nz=768, faces="z", nof=300, steps=128,
             block=128, structure="slit", ipol=2, kx=0.0, fields=1, plane=2),
        # the same grating in FP64, the reference's precision
        dict(name="slit_256x4x768_fp64", kind="engine", prec=64, nx=256, ny=4, nz=768, faces="z", nof=300, steps=64,
             block=32, structure="slit", ipol=2, kx=0.0, fields=1, plane=2),
        # a small unit cell of odd sizes at oblique Bloch phase with an absorbing structure, every face pair of the
        # DFT box as the reference accumulates them
        dict(name="cell_61x47x203_lossy_fp32", kind="engine", prec=32, nx=61, ny=47, nz=203, faces="all", nof=96,
             steps=64, block=64, structure="lossy", ipol=1, kx=0.3, fields=1, plane=3),
        # a mid-size cell (the gradient workload's grid), forward only
        dict(name="cell_160x160x512_fp32", kind="engine", prec=32, nx=160, ny=160, nz=512, faces="z", nof=64, steps=32,
             block=32, structure="pattern", ipol=2, kx=0.0, fields=1, plane=3),
        # the DFT-heavy form: every face pair of a 256x256x96 cell at 128 frequencies, a block committed in the pass
        dict(name="faces_256x256x96_nof128_fp32", kind="engine", prec=32, nx=256, ny=256, nz=96, faces="all", nof=128,
             steps=64, block=64, structure="spheres", ipol=2, kx=0.3, fields=1, plane=3),
        # the large 3D cell of the benchmark: 512x512x1024, Bloch phase 0.3 pi a cell, 200 spheres
        dict(name="spheres_512x512x1024_fp32", kind="engine", prec=32, nx=512, ny=512, nz=1024, faces="z", nof=100,
             steps=8, block=8, structure="spheres", ipol=2, kx=0.3, fields=0, plane=0),
        # the reference's own precision on a 3D cell with every face pair: what the drop-in program runs by default
        dict(name="spheres_128x128x160_fp64", kind="engine", prec=64, nx=128, ny=128, nz=160, faces="all", nof=128,
             steps=32, block=32, structure="spheres", ipol=2, kx=0.3, fields=1, plane=3),
        # the batched form: uneven unit cells (32..160 a side, 256..768 deep) stepped together, tuned once
        dict(name="batch_32cells_fp32", kind="batch", cells=32, nof=128, steps=8),
        # the gradient: forward and backward through the torch function, checkpointed and recomputed
        dict(name="adjoint_160x160x352_fp32", kind="adjoint", nx=160, ny=160, nz=352, dx=128, dy=128, dh=16, nof=64,
             steps=192, every=96),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["engine32", "engine32", "engine32", "engine64", "engine64", "batch", "adjoint", "deck"])
    if kind == "deck":
        nx = rng.choice([1, 1, _log(rng, 24, 120)])
        return dict(kind="deck", nx=nx, ny=1, nz=rng.randint(260, 520), pml=rng.randint(40, 75),
                    nof=rng.randint(50, 500), steps=rng.randint(300, 1200), outputs=rng.randint(1, 4))
    if kind == "batch":
        return dict(kind="batch", cells=rng.randint(4, 28), nof=rng.randint(32, 128), steps=8)
    if kind == "adjoint":
        nx, ny, nz = rng.randint(40, 150), rng.randint(40, 150), rng.randint(120, 340)
        return dict(kind="adjoint", nx=nx, ny=ny, nz=nz, dx=rng.randint(8, nx - 8), dy=rng.randint(8, ny - 8),
                    dh=rng.randint(4, 16), nof=rng.randint(8, 64), steps=rng.randint(120, 190),
                    every=rng.choice([48, 96, 200]))
    prec = 64 if kind == "engine64" else 32
    shape = rng.choice(["thin", "cube", "cube"])
    while True:
        if shape == "thin":
            nx, ny, nz = _log(rng, 2, 1024), rng.randint(1, 12), _log(rng, 128, 1024)
        else:
            nx, ny, nz = _log(rng, 16, 320), _log(rng, 16, 320), _log(rng, 64, 512)
        cells = nx * ny * nz
        if cells <= (2.5e6 if prec == 64 else 16e6):
            break
    steps = max(8, min(128, int((3e7 if prec == 64 else 3e8) / cells)))
    block = min(steps, 32) if prec == 64 else steps
    return dict(kind="engine", prec=prec, nx=nx, ny=ny, nz=nz, faces=rng.choice(["z", "z", "all"]),
                nof=rng.randint(16, 128), steps=steps, block=block,
                structure=rng.choice(["slab", "pattern", "spheres", "lossy"]), ipol=rng.choice([1, 2]),
                kx=rng.choice([0.0, round(rng.uniform(0.05, 0.5), 3)]), fields=1, plane=rng.choice([2, 3]))


# ---------------------------------------------------------------------------
# geometry and inputs

IT0 = 160  # the pulse passes the source plane around this step


def _layout(case):
    """UPML thickness, source plane, DFT planes and structure of one cell."""
    nz = case["nz"]
    pml = 16 if nz >= 256 else max(4, nz // 12)
    tfsf = pml + max(4, nz // 24)
    dh = max(2, nz // 6)
    hi = max(tfsf + 4, nz // 2 - dh // 2)
    return pml, tfsf, hi, dh


def _params(w, **over):
    d = tempfile.mkdtemp(prefix="iris_case_")
    try:
        p, fw, _ = iris.setparam(cfg.write_input(os.path.join(d, "inputFDTD.dat"), w, **over))
    finally:
        shutil.rmtree(d, ignore_errors=True)
    return p, fw


def _engine_setup(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    pml, tfsf, hi, dh = _layout(case)
    # with no wave in the cell yet, the reflection plane sits in the incident field just above the source
    r = (pml + tfsf) // 2 if case["fields"] else tfsf + 2
    box = (1, nx, 1, ny, r, nz - (pml + tfsf) // 2)
    if case["structure"] == "slit":
        w = cfg.Workload("c", nx, ny, nz, pml, nz + 1 - pml, hi, dh, 4.0, max(1, nx // 4), tfsf, box, case["nof"],
                         case["steps"], structure="slit")
    else:
        w = cfg.Workload("c", nx, ny, nz, pml, nz + 1 - pml, hi, dh, 2.25 if case["structure"] == "slab" else 1.0, 0,
                         tfsf, box, case["nof"], case["steps"])
    p, fw = _params(w, i_pol=case["ipol"])
    p.akx_re = case["kx"] * math.pi * nx
    p.epump *= float(np.random.default_rng(seed + 5).uniform(0.5, 2.0))
    if case["faces"] == "z":
        p.dft_faces = iris.DFT_Z
    return w, p, fw


def _spheres(case, w, seed):
    r = np.random.default_rng(seed)
    n = 200 if w.cells > 10 ** 7 else 24
    big = max(2.0, min(32.0, min(w.nx, w.ny, w.dh) / 3.0))
    hf = w.hi + w.dh - 1
    return np.stack([r.uniform(1, w.nx, n), r.uniform(1, w.ny, n), r.uniform(w.hi, hf, n),
                     r.uniform(big / 4, big, n), r.uniform(1.5, 6.0, n)], axis=1)


def _material(case, w, seed):
    """eps_inv planes hi-1..hf+1 for structures uploaded from the host."""
    a = cfg.slit_material(w)
    r = np.random.default_rng(seed)
    if case["structure"] in ("slab", "slit"):
        a[1:-1] = np.where(a[1:-1] == 1.0, 1.0, 1.0 / r.uniform(2.0, 9.0))
    else:  # weakly absorbing blocks (a scalar complex eps_inv amplifies one sign of frequency: kept small)
        eps = r.uniform(1.5, 6.0, a[1:-1].shape[0]) + 1j * r.uniform(1e-6, 5e-6, a[1:-1].shape[0])
        a[1:-1] = (1.0 / eps)[:, None, None]
        n = max(1, w.nx // 2)
        a[1:-1, :, 1:1 + n] = 1.0
        cfg._wrap_ghosts(a)
    return a


def _fields(case, p, seed):
    """A wave in the cell: a few Bloch modes of random amplitude, zero in the UPML slabs; E and H as complex
    [z, y, x, c] over 0..n+1 on the GPU."""
    nx, ny, nz = p.nx, p.ny, p.nz
    r = np.random.default_rng(seed + 17)
    dev = "cuda"

    def axis(n, k):
        return torch.exp(1j * k * torch.arange(n + 2, dtype=torch.float64, device=dev))

    z = np.arange(nz + 2)
    t = np.clip((z - p.pmlzi) / max(1.0, p.pmlzf - p.pmlzi), 0.0, 1.0)
    win = torch.from_numpy(np.sin(np.pi * t) ** 2).to(dev)
    win[: p.pmlzi + 1] = 0.0
    win[p.pmlzf:] = 0.0
    out = []
    for scale in (1.0, 0.3):
        f = torch.zeros((nz + 2, ny + 2, nx + 2, 3), dtype=torch.complex128, device=dev)
        for _ in range(3):
            mx, my = int(r.integers(-2, 3)), int(r.integers(-2, 3))
            amp = torch.from_numpy(r.normal(size=3) + 1j * r.normal(size=3)).to(dev) * (p.epump * p.Q * scale)
            ez = axis(nz, r.uniform(-0.6, 0.6)) * win
            ey = axis(ny, 2 * math.pi * my / ny)
            ex = axis(nx, (2 * math.pi * mx + p.akx_re) / nx)
            f += (ez[:, None] * ey)[:, :, None, None] * (ex[:, None] * amp)
        out.append(f)
    return out


def _batch_setup(case, seed):
    ws = cfg.batch_cells(case["cells"], seed=0, nof=case["nof"], nsteps=case["steps"])
    ps = []
    for w in ws:
        w.box = (1, w.nx, 1, w.ny, w.tfsf_zi + 2, w.tfsf_zi + 8)
        p, fw = _params(w)
        p.dft_block = case["steps"]
        ps.append(p)
    fill = np.random.default_rng(seed).uniform(0.3, 0.7, len(ws))
    amp = np.random.default_rng(seed + 1).uniform(0.5, 2.0, len(ws))
    for p, a in zip(ps, amp):
        p.epump *= a
    return ws, ps, fw, fill


BATCH_WARM = 40  # steps from the pulse's arrival to the first pass


def _adjoint_setup(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    pml, tfsf, hi = 12, 16, 22
    t = hi + case["dh"] + 6
    w = cfg.Workload("a", nx, ny, nz, pml, nz + 1 - pml, hi, case["dh"], 1.0, 0, tfsf, (1, nx, 1, ny, 14, t),
                     case["nof"], case["steps"])
    p, fw = _params(w, pulse_steps=20.0)
    x0, y0 = (nx - case["dx"]) // 2 + 1, (ny - case["dy"]) // 2 + 1
    design = (x0, x0 + case["dx"] - 1, y0, y0 + case["dy"] - 1, hi, hi + case["dh"] - 1)
    shape = (case["dh"], case["dy"], case["dx"])
    eps = 1.0 + 3.0 * np.random.default_rng(seed).random(shape)
    return w, p, fw, design, eps


def _deck(case, d, seed):
    nx, nz, pml = case["nx"], case["nz"], case["pml"]
    tfsf = pml + 12
    hi = nz // 2 - 15
    w = cfg.Workload("deck", nx, case["ny"], nz, pml, nz + 1 - pml, hi, 30,
                     float(np.random.default_rng(seed).uniform(2.0, 9.0)), 0 if nx == 1 else max(1, nx // 5), tfsf,
                     (1, nx, 1, case["ny"], pml + 6, nz - pml - 6), case["nof"], case["steps"])
    kw = dict(no_downloads=case["outputs"], pulse_steps=60.0, wlpump=200.0, cfl=0.8, lno=120.0,
              dlamda=300.0 / case["nof"])
    return cfg.make_run(w, d, **kw)


class _RunDir:
    """A run directory, removed with the state that holds it."""

    def __init__(self):
        self.path = tempfile.mkdtemp(prefix="iris_deck_")

    def __del__(self):
        shutil.rmtree(self.path, ignore_errors=True)


# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "deck":
        d = _RunDir()
        _deck(case, d.path, seed)
        return dict(case=case, dir=d)
    if kind == "batch":
        ws, ps, fw, fill = _batch_setup(case, seed)
        b = iris.Batch(ps, fw, precision=iris.FP32, dft_faces=iris.DFT_Z, dft_block=case["steps"])
        for i, w in enumerate(ws):
            b.material_pattern(i, seed * 1000 + i, float(fill[i]))
        b.autotune()
        b.step(IT0, BATCH_WARM)
        return dict(case=case, b=b, it=IT0 + BATCH_WARM)
    if kind == "adjoint":
        w, p, fw, design, eps = _adjoint_setup(case, seed)
        adj = iris.Adjoint(p, fw, design, checkpoint_every=case["every"], precision=iris.FP32)
        return dict(case=case, adj=adj, f=iris.design_objective(adj, case["steps"]),
                    eps=torch.from_numpy(eps).to("cuda", torch.float32).requires_grad_(True))
    w, p, fw = _engine_setup(case, seed)
    e = iris.Engine(p, fw, precision=iris.FP64 if case["prec"] == 64 else iris.FP32, dft_block=case["block"])
    if case["structure"] == "spheres":
        e.material_spheres(_spheres(case, w, seed))
    elif case["structure"] == "pattern":
        e.material_pattern(seed, 0.5)
    else:
        e.set_material(_material(case, w, seed))
    if case["fields"]:
        for which, f in zip((iris.E, iris.H), _fields(case, e.p, seed)):
            e.set_field_c(which, f.cpu().numpy())
    return dict(case=case, e=e, it=IT0)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "deck":
        d = state["dir"].path
        names = [os.path.join(d, "1_scatt%s.dat" % j) for j in ("5", "6")]
        for f in os.listdir(d):
            if f.startswith("1_scatt"):
                os.remove(os.path.join(d, f))
        iris.run_input(d, iris.FP64)
        return [iris.read_scatt(f, case["nof"]) for f in names]
    n = case["steps"]
    if kind == "batch":
        b = state["b"]
        b.step(state["it"], n)
        state["it"] += n
        return [b.flux(i).astype(np.float32) for i in range(b.n)]
    if kind == "adjoint":
        eps = state["eps"]
        eps.grad = None
        L = state["f"](eps)
        L.backward()
        return [np.float32(float(L)), eps.grad]
    e = state["e"]
    e.step(state["it"], n)
    state["it"] += n
    J = e.flux(0)
    out = [J]
    p = e.p
    if case["plane"] == 2:
        y = (p.ny + 1) // 2
        out.append(e.get_plane(iris.E, 2, y, (1, p.nx), (1, p.nz)))
    elif case["plane"] == 3:
        out.append(e.get_plane(iris.H, 3, p.nz // 2, (1, p.nx), (1, p.ny)))
    elif case["fields"]:
        out += [e.get_field_c(iris.E), e.get_field_c(iris.H)]
    if case["prec"] == 32:
        out = [a.astype(np.complex64 if np.iscomplexobj(a) else np.float32) for a in out]
    return out


# ---------------------------------------------------------------------------

def _step_work(cells, upml_cells, s):
    """Bytes of one state of complex values of s bytes (E, H; D, B in the slabs), and one step's operations."""
    return (6 * cells + 6 * upml_cells) * s, 60 * cells + 96 * upml_cells


def _dft_points(nx, ny, nz, box, faces):
    n = 12 * (box[1] - box[0] + 1) * (box[3] - box[2] + 1)
    if faces == "all":
        n += 12 * (box[5] - box[4] + 1) * ((box[1] - box[0] + 1) + (box[3] - box[2] + 1))
    return n


def _engine_work(cells, upml, s, steps, points, nof):
    state, ops = _step_work(cells, upml, s)
    by = 2 * state * (1 if state < ON_CHIP_BYTES else steps)
    return by + 32 * points * nof, steps * (ops + 8.0 * points * nof)


def work(case):
    kind = case["kind"]
    if kind == "deck":
        cells = case["nx"] * case["ny"] * case["nz"]
        b, f = _engine_work(cells, cells * 2 * case["pml"] // case["nz"], 16, case["steps"], 12 * case["nx"], case["nof"])
    elif kind == "batch":
        b = f = 0.0
        for w in cfg.batch_cells(case["cells"], nof=case["nof"]):
            state, ops = _step_work(w.cells, w.nx * w.ny * 32, 8)
            points = 12 * w.nx * w.ny
            b += 2 * state * case["steps"] + 32 * points * case["nof"]
            f += case["steps"] * (ops + 8.0 * points * case["nof"])
    elif kind == "adjoint":
        cells = case["nx"] * case["ny"] * case["nz"]
        state, ops = _step_work(cells, case["nx"] * case["ny"] * 24, 8)
        rec = 2 * 24 * case["dx"] * case["dy"] * case["dh"]  # the design cells' curls, written and read
        points = 12 * case["nx"] * case["ny"]
        b = case["steps"] * (4 * state + rec) + 32 * points * case["nof"]
        f = case["steps"] * 2.0 * (ops + 8.0 * points * case["nof"])
    else:
        pml, tfsf, hi, dh = _layout(case)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        points = _dft_points(nx, ny, nz, (1, nx, 1, ny, (pml + tfsf) // 2, nz - (pml + tfsf) // 2), case["faces"])
        b, f = _engine_work(nx * ny * nz, nx * ny * 2 * pml, case["prec"] // 4, case["steps"], points, case["nof"])
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, by whole-array torch operations

class _Plain:
    """The time loop of the reference (code/driver.f90:338-451) on complex128 arrays [c][z, y, x] over 0..n+1."""

    def __init__(self, p, fw, eps_inv, e=None, h=None):
        self.p, self.fw, dev = p, np.asarray(fw), "cuda"
        self.dev = dev
        shape = (p.nz + 2, p.ny + 2, p.nx + 2)
        mk = lambda f: ([f[..., c].contiguous() for c in range(3)] if f is not None  # noqa: E731
                        else [torch.zeros(shape, dtype=torch.complex128, device=dev) for _ in range(3)])
        self.E, self.H = mk(e), mk(h)
        self.slabs = [(1, p.pmlzi, p.eps1), (p.pmlzf, p.nz, p.eps3)]
        z = lambda lo, hi: torch.zeros((hi - lo + 1, p.ny, p.nx), dtype=torch.complex128, device=dev)  # noqa: E731
        self.D = [[z(lo, hi) for _ in range(3)] for lo, hi, _ in self.slabs]
        self.B = [[z(lo, hi) for _ in range(3)] for lo, hi, _ in self.slabs]
        self.cf = [self._rows(s) for s in range(2)]
        m = torch.full((p.nz + 2, 1, 1), 1.0 / p.eps1, dtype=torch.float64, device=dev)
        m[p.hf + 1:] = 1.0 / p.eps3
        self.m = m
        self.eps = eps_inv  # planes hi..hf, interior cells, or None
        dtc = p.dt * p.c0 / p.Q
        self.dtcq2 = dtc * dtc
        self.ph = [np.exp(1j * complex(a, b)) for a, b in ((p.akx_re, p.akx_im), (p.aky_re, p.aky_im), (p.akz_re, p.akz_im))]
        self.mh = [np.exp(-1j * complex(a, b)) for a, b in ((p.akx_re, p.akx_im), (p.aky_re, p.aky_im), (p.akz_re, p.akz_im))]
        self.samples, self.times = {}, []

    def _rows(self, s):
        p = self.p
        lo, hi, epsb = self.slabs[s]
        z = np.arange(lo, hi + 1, dtype=np.float64)
        g = ((p.pmlzi - z) / (p.pmlzi - 1.0)) ** p.npml if s == 0 else ((z - p.pmlzf) / (p.nz - p.pmlzf)) ** p.npml
        sg, kk = math.sqrt(epsb) * p.wzpml * g, 1.0 + math.sqrt(epsb) * p.pmlalfa * g
        one = np.ones_like(z)
        fp = [2 * p.eps0 * epsb * one, 2 * p.eps0 * epsb * one, 2 * p.eps0 * epsb * kk + p.dt * sg]
        fm = [2 * p.eps0 * epsb * one, 2 * p.eps0 * epsb * one, 2 * p.eps0 * epsb * kk - p.dt * sg]
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)[:, None, None]  # noqa: E731
        out = []
        for k in range(3):
            d, e = (k + 1) % 3, (k + 2) % 3
            out.append(dict(a=t(fm[d] / fp[d]), b=t(2 * epsb / fp[d]), ea=t(fm[e] / fp[e]),
                            eb=t(1 / (p.eps0 * epsb * fp[e])), fp=t(fp[k]), fm=t(fm[k]),
                            bb=t(2 * epsb / fp[d] * (p.dt / p.Q) ** 2), hb=t(1 / (p.mu0 * fp[e]))))
        return out

    def step(self, it, sample):
        p, E, H = self.p, self.E, self.H
        X, Y, Z = slice(1, p.nx + 1), slice(1, p.ny + 1), slice(1, p.nz + 1)
        xm, ym, zm = slice(0, p.nx), slice(0, p.ny), slice(0, p.nz)
        xp, yp, zp = slice(2, p.nx + 2), slice(2, p.ny + 2), slice(2, p.nz + 2)
        for k in range(3):
            i, j = (k + 1) % 3, (k + 2) % 3
            # E_k += curl: d H_j along axis i minus d H_i along axis j (axes x, y, z = 0, 1, 2)
            sel = lambda ax: ((Z, Y, xm), (Z, ym, X), (zm, Y, X))[ax]  # noqa: E731
            c = (H[j][Z, Y, X] - H[j][sel(i)]) - (H[i][Z, Y, X] - H[i][sel(j)])
            new = E[k][Z, Y, X] + self.m[1:-1] * c
            if self.eps is not None and p.hf >= p.hi:
                q = slice(p.hi - 1, p.hf)
                new[q] = E[k][p.hi:p.hf + 1, Y, X] + self.eps * c[q]
            for s, (lo, hi, _) in enumerate(self.slabs):
                q, cf = slice(lo - 1, hi), self.cf[s][k]
                d0 = self.D[s][k]
                d1 = cf["a"] * d0 + cf["b"] * (p.eps0 ** 2 * c[q])
                self.D[s][k] = d1
                new[q] = cf["ea"] * E[k][lo:hi + 1, Y, X] + cf["eb"] * (cf["fp"] * d1 - cf["fm"] * d0)
            E[k][Z, Y, X] = new
        for k in range(3):
            E[k][Z, Y, p.nx + 1] = self.ph[0] * E[k][Z, Y, 1]
            E[k][Z, p.ny + 1, X] = self.ph[1] * E[k][Z, 1, X]
            E[k][p.nz + 1, Y, X] = self.ph[2] * E[k][1, Y, X]
        for k in range(3):
            i, j = (k + 1) % 3, (k + 2) % 3
            sel = lambda ax: ((Z, Y, xp), (Z, yp, X), (zp, Y, X))[ax]  # noqa: E731
            c = (E[j][sel(i)] - E[j][Z, Y, X]) - (E[i][sel(j)] - E[i][Z, Y, X])
            new = H[k][Z, Y, X] - self.dtcq2 * c
            for s, (lo, hi, _) in enumerate(self.slabs):
                q, cf = slice(lo - 1, hi), self.cf[s][k]
                b0 = self.B[s][k]
                b1 = cf["a"] * b0 - cf["bb"] * c[q]
                self.B[s][k] = b1
                new[q] = cf["ea"] * H[k][lo:hi + 1, Y, X] + cf["hb"] * (cf["fp"] * b1 - cf["fm"] * b0)
            H[k][Z, Y, X] = new
        for F in (E, H):
            for k in range(3):
                F[k][Z, Y, 0] = self.mh[0] * F[k][Z, Y, p.nx]
                F[k][Z, 0, X] = self.mh[1] * F[k][Z, p.ny, X]
                F[k][0, Y, X] = self.mh[2] * F[k][p.nz, Y, X]
        self._source(it)
        if sample:
            self.times.append(it + 1 - p.to_fourier)
            for f, (comps, at) in self._faces().items():
                self.samples.setdefault(f, []).append([(E[c] if c < 3 else H[c - 3])[at].reshape(-1).clone() for c in comps])

    def _incident(self, iz, it):
        """tf1/tf5 (or tf2/tf4) of the Gaussian pulse at plane iz over ix = 0..nx+1."""
        p = self.p
        eps_s, sk = (p.eps3, -1.0) if p.tfsf_zi > p.hi else (p.eps1, 1.0)
        delta = p.ratio_angle * p.pi / 2.0
        ux, uz = math.cos(delta), math.sin(delta)
        ix = np.arange(p.nx + 2)
        t = p.c0 * p.dt * it
        A = p.Q * (ix - (p.pmlzi - 50)) * ux + p.Q * (iz - p.zopump) * uz
        env = np.exp(-(((A - t / math.sqrt(eps_s)) / (p.gpump * p.Q)) ** 2))
        ko = 2 * p.pi / (p.wlpump * p.f_abohr)
        w = env * np.exp(1j * ko * (math.sqrt(eps_s) * sk * A - t))
        amp, hc = p.epump * p.Q, p.epump * p.Q * (p.dt * p.c0 / p.Q)
        if p.i_pol == 2:
            ex, ez = uz * sk * w, -ux * w
            return amp * ex, hc * (uz * sk * ex - ux * ez), eps_s
        hx, hz = -uz * sk * w, ux * w
        return amp * (ux * hz - uz * sk * hx), hc * hx, eps_s

    def _source(self, it):
        p, zm = self.p, self.p.tfsf_zi
        three = p.nx != 1 and p.ny != 1
        t = lambda a: torch.from_numpy(a).to(self.dev)[None, :]  # noqa: E731
        if three or p.i_pol == 1:
            vE, vH = t(self._incident(zm - 1, it)[1] / p.eps1), t(self.dtcq2 * self._incident(zm, it)[0])
            if p.i_pol == 2:
                self.E[0][zm, :, :p.nx + 1] += vE[:, :p.nx + 1]
                self.H[1][zm - 1, :, :p.nx + 1] += vH[:, :p.nx + 1]
            else:
                self.E[1][zm, :p.ny + 1] -= vE
                self.H[0][zm - 1, :p.ny + 1] -= vH
        else:
            a, b, eps_s = self._incident(zm, it)
            self.E[0][zm] += t(b / eps_s)
            self.H[1][zm] += t(self.dtcq2 * a)

    def _faces(self):
        p, out = self.p, {}
        bx = [p.box1[i] for i in range(6)]
        x, y, z = (slice(bx[2 * i], bx[2 * i + 1] + 1) for i in range(3))
        if p.dft_faces == iris.DFT_Z:
            on = (False, False, True)
        elif p.nx != 1 and p.ny != 1:
            on = (True, True, True)
        else:
            on = (p.ny == 1 and p.nx != 1, p.nx == 1 and p.ny != 1, True)
        comps = ((1, 5, 2, 4), (2, 3, 0, 5), (0, 4, 1, 3))
        for j in range(3):
            if on[j]:
                for side in range(2):
                    at = bx[2 * j + side]
                    out[2 * j + side] = (comps[j], ((z, y, at), (z, at, x), (at, y, x))[j])
        return out

    def flux(self):
        p = self.p
        J = np.zeros((6, p.nof))
        W = torch.from_numpy(p.dt * np.exp(1j * np.outer(self.fw, np.asarray(self.times, dtype=np.float64)))).to(self.dev)
        for f, s in self.samples.items():
            n = s[0][0].numel()
            tot = torch.zeros(p.nof, dtype=torch.float64, device=self.dev)
            for q in range(0, n, 1 << 16):
                A = [W @ torch.stack([x[c][q:q + (1 << 16)] for x in s]) for c in range(4)]
                tot += ((A[0] * A[1].conj()).real - (A[2] * A[3].conj()).real).sum(1)
            J[f] = (1 if f % 2 else -1) * p.eps0 * p.Q / (2 * p.dt) * tot.cpu().numpy()
        return J


def _exact_material(case, w, seed):
    s = case["structure"]
    w.extra = dict(seed=seed)
    if s == "spheres":
        # the voxeliser's rule (later spheres win, periodic in x and y) over whole bounding boxes
        a = torch.ones((w.dh, w.ny, w.nx), dtype=torch.float64, device="cuda") / w.eps_bbox
        hf = w.hi + w.dh - 1
        ar = lambda lo, hi: torch.arange(lo, hi + 1, device="cuda")  # noqa: E731
        for cx, cy, cz, rad, eps in _spheres(case, w, seed):
            z = ar(max(w.hi, math.floor(cz - rad)), min(hf, math.ceil(cz + rad)))
            y = ar(math.floor(cy - rad), math.ceil(cy + rad))[: w.ny]
            x = ar(math.floor(cx - rad), math.ceil(cx + rad))[: w.nx]
            inside = ((z[:, None, None] - cz) ** 2 + (y[None, :, None] - cy) ** 2 + (x[None, None, :] - cx) ** 2) <= rad * rad
            at = ((z - w.hi)[:, None, None], ((y - 1) % w.ny)[None, :, None], ((x - 1) % w.nx)[None, None, :])
            a[at] = torch.where(inside, torch.full_like(a[at], 1.0 / eps), a[at])
        return a
    if s == "pattern":
        u = cfg.splitmix_uniform(seed, np.arange(w.dh * w.ny * w.nx)).reshape(w.dh, w.ny, w.nx)
        return torch.from_numpy(np.where(u < 0.5, 0.25, 1.0)).to("cuda")
    return torch.from_numpy(np.ascontiguousarray(_material(case, w, seed)[1:-1, 1:-1, 1:-1])).to("cuda")


def exact(case, seed):
    kind = case["kind"]
    if kind == "deck":
        d = _RunDir()
        p, fw, _ = iris.setparam(_deck(case, d.path, seed))
        a = iris.set_emconstants(p)[1:-1, 1:-1, 1:-1]
        s = _Plain(p, fw, torch.from_numpy(np.ascontiguousarray(a)).to("cuda"))
        out, nos = [], 1
        for it in range(1, p.texit + 1):
            s.step(it, True)
            if it == p.no_downloads * nos or it == p.texit:
                nos += 1
                out.append(s.flux())
        return [np.stack([J[4] for J in out]), np.stack([J[5] for J in out])]
    if kind == "batch":
        ws, ps, fw, fill = _batch_setup(case, seed)
        out = []
        for i, (w, p) in enumerate(zip(ws, ps)):
            p.dft_faces = iris.DFT_Z
            u = cfg.splitmix_uniform(seed * 1000 + i, np.arange(w.dh * w.ny * w.nx)).reshape(w.dh, w.ny, w.nx)
            s = _Plain(p, fw, torch.from_numpy(np.where(u < float(fill[i]), 0.25, 1.0)).to("cuda"))
            for it in range(IT0, IT0 + BATCH_WARM + case["steps"]):
                s.step(it, True)
            out.append(s.flux())
            del s
        return out
    if kind == "adjoint":
        w, p, fw, design, eps = _adjoint_setup(case, seed)
        p.dft_faces = iris.DFT_Z
        m = torch.ones((w.dh, w.ny, w.nx), dtype=torch.float64, device="cuda")
        x0, x1, y0, y1, _, _ = design
        m[:, y0 - 1:y1, x0 - 1:x1] = 1.0 / torch.from_numpy(eps.astype(np.float32).astype(np.float64)).to("cuda")
        s = _Plain(p, fw, m)
        for it in range(1, case["steps"] + 1):
            s.step(it, True)
        return [float(s.flux()[5].sum()), None]
    w, p, fw = _engine_setup(case, seed)
    e = h = None
    if case["fields"]:
        e, h = _fields(case, p, seed)
        if case["prec"] == 32:
            e, h = (f.to(torch.complex64).to(torch.complex128) for f in (e, h))
    s = _Plain(p, fw, _exact_material(case, w, seed), e, h)
    for it in range(IT0, IT0 + case["steps"]):
        s.step(it, True)
    out = [s.flux()]
    if case["plane"] == 2:
        y = (p.ny + 1) // 2
        out.append(torch.stack([s.E[c][1:p.nz + 1, y, 1:p.nx + 1] for c in range(3)], dim=-1))
    elif case["plane"] == 3:
        out.append(torch.stack([s.H[c][p.nz // 2, 1:p.ny + 1, 1:p.nx + 1] for c in range(3)], dim=-1))
    elif case["fields"]:
        out += [torch.stack(s.E, dim=-1), None]  # H's ghost planes at n+1 hold no value of the time loop
    return out
