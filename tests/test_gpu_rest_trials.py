"""Obstacles placed after the trial steps of Batch.autotune: the trials write both
population buffers and leave the step count where it was, so the new obstacles
do not start at rest in the buffer the first step writes."""
import numpy as np
import pytest

from fluidmaxxer_b200 import lattice

from .test_gpu_rest_obstacles import KEYS, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["mask", "bits"])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_obstacles_placed_after_autotune(prec, how):
    p = problem(96)
    solid = p.solid.reshape(p.nz, p.ny, p.nx).copy()
    solid[3:6, 3:9, 30:62] = 1
    solid = solid.reshape(-1)
    tuned, fresh = lattice.from_problem(p, prec), lattice.from_problem(p, prec)
    B = lattice.Batch([tuned])
    B.autotune(trial_steps=4)
    B.close()
    assert tuned.step_count == 0
    for L in (tuned, fresh):
        if how == "mask":
            L.set_obstacle_mask(solid)
        else:
            L.set_obstacle_bits(np.packbits(solid, bitorder="little").view(np.uint32))
    for steps in (1, 1, 1, 8):
        for L in (tuned, fresh):
            L.step(steps)
        got, ref = tuned.get_state(), fresh.get_state()
        for k in KEYS:
            assert np.array_equal(got[k], ref[k]), (k, steps)
    for L in (tuned, fresh):
        L.close()
