"""The FP32 gradient's DFT sources, formed for a block of sampled steps at a
time in integers: blocks of 64 steps and a remainder, one frequency and
more than a warp of them, every sampling interval, both faces with weights far
apart, points that do not fill a block.  FP32 against FP64, with the tolerance
of the FP32 gradient (1e-3 of the largest entry: the fields' own rounding over
hundreds of steps)."""
import numpy as np
import pytest

from test_gpu_adjoint import gradient, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nof,every,nsteps", [(1, 1, 331), (33, 3, 600), (6, 7, 450), (6, 1, 515)])
def test_block_sources_match_fp64(iris, tmp_path, nof, every, nsteps):
    p, fw, eps_inv, eta = small_case(iris, tmp_path, nsteps=nsteps, nof=nof)
    p.sample_fourier = every
    r = np.random.default_rng(2)
    weights = (r.uniform(-1e-6, 1e-6, nof), r.uniform(0.5, 1.5, nof))
    _, L64, _, g64 = gradient(iris, p, fw, eps_inv, eta, 0, weights=weights, nsteps=nsteps)
    _, L32, _, g32 = gradient(iris, p, fw, eps_inv, eta, 1, weights=weights, nsteps=nsteps)
    assert abs(L32 - L64) <= 1e-4 * abs(L64)
    assert np.max(np.abs(g32 - g64)) <= 1e-3 * np.max(np.abs(g64))
