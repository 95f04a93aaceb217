"""The resident kernel's packet exchange (FP64 grids whose CTAs take a phase in
one round): bit for bit the split passes, with phases on y and z (both parts of
a neighbour's value), complex materials, fewer rows than SMs, rows whose y
neighbours are other CTAs', the largest CTA it takes, one step a launch and
launches that follow one another."""
import numpy as np
import pytest

import test_gpu_resident as resident

pytestmark = pytest.mark.gpu

# as resident.CASES
CASES = {
    "phases_everywhere": (4, 3, 64, 5, 12, 2, (0.3, -0.7, 0.4), False, 9),
    "phases_lossy": (4, 3, 64, 5, 12, 2, (0.3, -0.7, 0.4), True, 9),
    "one_column_z_phase": (1, 1, 300, 20, 40, 2, (0, 0, 0.4), True, 9),
    "one_row_a_cta": (20, 1, 100, 8, 20, 1, (0.2, 0, 0), False, 8),
    "many_y": (2, 60, 20, 4, 8, 2, (0.3, 0.5, 0), True, 7),
    "largest": (85, 1, 150, 10, 30, 2, (0.3, 0, 0.2), False, 7),
    "one_step": (4, 4, 100, 8, 20, 2, (0.3, 0.2, 0.1), False, 1),
}


@pytest.mark.parametrize("name", CASES)
def test_packets_equal_split(iris, tmp_path, monkeypatch, name):
    monkeypatch.setattr(resident, "CASES", CASES)
    resident.test_resident_equals_split(iris, tmp_path, name, iris.FP64)
