"""bench.py's roofline counts the bytes a step moves: the populations of resting
obstacles, which the FP32 and FP64 steps leave out, are not among them."""
import os
import sys

import numpy as np
import pytest

from fluidmaxxer_b200 import problems

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.parametrize("prec,sector", [("f32", 8), ("f64", 4)])
@pytest.mark.parametrize("nx", [16, 33, 40])
def test_resting_cells_by_hand(nx, prec, sector):
    ny, nz = 7, 6
    solid = (np.random.default_rng(nx).random((nz, ny, nx)) < 0.9).astype(np.uint8).reshape(-1)
    p = problems.Problem(nx=nx, ny=ny, nz=nz, solid=solid, tau=0.7, tau_ad=0.6, u_in=(0.01, 0.0, 0.0))
    want = 0
    for c in range(nx * ny * nz):
        first = c - c % sector
        cells = range(first, first + sector)
        if cells[-1] >= solid.size or any(not solid[k] for k in cells):
            continue
        x = c % nx - c % sector
        want += x >= 2 and x + sector - 1 <= nx - 3
    assert bench.resting_cells(p, prec) == want
    assert bench.step_bytes(p, prec) == bench.BYTES_PER_CELL[prec] * p.n_cells - 38 * (32 // sector) * want
    assert bench.step_bytes(p, prec, rest=False) == bench.BYTES_PER_CELL[prec] * p.n_cells
    assert bench.resting_cells(p, "f16") == 0
