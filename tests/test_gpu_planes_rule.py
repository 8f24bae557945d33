"""The step takes its boundary planes from the boundary cells' inward neighbours or
from the boundary cells' own lanes, by storage type, row length, lattice size
and whether the step's outputs may be read: within one call the last step can
differ from the others.  Monitored steps always take the lanes, so a lattice
that alternates has to end up as one that is monitored on every step."""
import numpy as np
import pytest

from fluidmaxxer_b200 import lattice, problems

pytestmark = pytest.mark.gpu


# sizes where a call of one step, the last step of a call or every step takes the lanes, and ones just inside each line
@pytest.mark.parametrize("prec,size", [("f32", (46, 276, 275)), ("f32", (46, 276, 276)), ("f32", (48, 260, 258)),
                                       ("f32", (62, 232, 232)), ("f32", (62, 232, 234)), ("f16", (190, 172, 175)),
                                       ("f16", (190, 176, 180)), ("f16", (192, 204, 204)), ("f16", (192, 204, 205)),
                                       ("f16", (64, 176, 178)), ("f16q", (64, 176, 178)), ("f16q", (448, 140, 130)),
                                       ("bf16", (96, 120, 124)), ("bf16", (96, 120, 126)), ("bf16", (190, 168, 170)),
                                       ("f16", (448, 232, 231))])
def test_same_state_as_monitored_steps(prec, size):
    p = problems.channel_small(11, *size)
    a, b = lattice.from_problem(p, prec), lattice.from_problem(p, prec)
    b.set_monitor(1)
    for steps in (1, 3, 2):
        a.step(steps)
        b.step(steps)
        got, ref = a.fields(dtype=np.float32), b.fields(dtype=np.float32)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (k, steps)
    if a.n < 9000000:   # populations come as doubles
        got, ref = a.get_state(), b.get_state()
        for k in ("f", "g", "phi", "q"):
            assert np.array_equal(got[k], ref[k]), k
    a.close()
    b.close()


def test_batch_equals_single_lattices():
    """Mode 3 of a batch takes the same rule: here only the steps whose outputs may
    be read, the last of a call or of a replayed graph, take the lanes."""
    sizes = [(64, 176, 178), (96, 176, 178)]
    solo = [lattice.from_problem(problems.channel_small(5, *s), "f16") for s in sizes]
    both = [lattice.from_problem(problems.channel_small(5, *s), "f16") for s in sizes]
    B = lattice.Batch(both)
    B.set_config(mode=3)
    for steps in (1, 5, 4):
        B.step(steps)
        B.synchronize()
        for a, b in zip(solo, both):
            a.step(steps)
            got, ref = b.fields(dtype=np.float32), a.fields(dtype=np.float32)
            for k in ref:
                assert np.array_equal(got[k], ref[k]), (k, steps)
    B.close()
    for L in solo + both:
        L.close()
