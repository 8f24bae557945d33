"""Boundary planes written by their inward neighbours (coupled_cell_direct):
row lengths around the warp size and the shortest rows that take it, so a warp
holds parts of one, two or three rows.  With odd row lengths a boundary cell
and its neighbour also fall into different warps and blocks."""
import dataclasses

import numpy as np
import pytest

from fluidmaxxer_b200 import lattice, problems, synth
from fluidmaxxer_b200._abi import FmError
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def problem(nx, collision="bgk"):
    ny, nz = 7, 6
    n = nx * ny * nz
    solid = synth.bernoulli(nx, ny, nz, 0.3, 1000 + nx, fluid_lo=0, fluid_hi=0, walls=True)
    more = {}
    if collision == "porous":
        r = np.random.default_rng(nx)
        more = dict(porosity=r.uniform(0.3, 1.0, n), region=(r.uniform(size=n) < 0.4).astype(np.uint8))
        solid = np.zeros(n, np.uint8)
    return problems.Problem(nx=nx, ny=ny, nz=nz, solid=solid, collision=collision, tau=0.7, tau_ad=0.6,
                            u_in=(0.02, 0.0, 0.0), isotherm="langmuir", q_max=3.0, b_langmuir=1.2, k_ldf=0.05,
                            **more)


# 14: the planes in the boundary cells' own lanes, 15: the boundary kernels over
# cell lists; 16 and 17: the shortest direct rows (two inlet rows a warp)
EVEN = [14, 16, 18, 30, 32, 34, 64, 96]
ODD = [15, 17, 19, 31, 33, 63, 65, 97]


@pytest.mark.parametrize("collision", ["bgk", "porous"])
@pytest.mark.parametrize("nx", EVEN + ODD)
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_bit_exact_vs_oracle(nx, collision, prec):
    p = problem(nx, collision)
    L = lattice.from_problem(p, prec)
    o = Oracle(p, "restated", prec)
    for steps in (1, 2, 40):
        L.step(steps)
        o.step(steps)
        got, ref = L.get_state(), o.get(populations=True)
        for k in ("f", "g", "phi", "q"):
            assert np.array_equal(got[k], ref[k]), (k, steps)
    L.close()
    o.close()


@pytest.mark.parametrize("collision", ["bgk", "porous"])
@pytest.mark.parametrize("nx", EVEN)
@pytest.mark.parametrize("prec", ["f16", "bf16", "f16q"])
def test_16_bit_equals_monitored_steps(nx, collision, prec):
    """Monitored steps keep the boundary planes in the boundary cells' own lanes."""
    p = problem(nx, collision)
    a, b = lattice.from_problem(p, prec), lattice.from_problem(p, prec)
    b.set_monitor(1)
    for steps in (1, 2, 40):
        a.step(steps)
        b.step(steps)
        got, ref = a.get_state(), b.get_state()
        for k in ("f", "g", "phi", "q"):
            assert np.array_equal(got[k], ref[k]), (k, steps)
    a.close()
    b.close()


def list_path(p, prec):
    """`p` with its pressure outlet added as two half planes, which runs every
    boundary as a kernel over a cell list."""
    half = np.zeros((p.nz, p.ny, p.nx), np.uint8)
    half[: p.nz // 2, :, -1] = 1
    rest = np.zeros_like(half)
    rest[p.nz // 2:, :, -1] = 1
    q = dataclasses.replace(p, ns_outlet="none")
    L = lattice.from_problem(q, prec)
    L.add_ns_pressure(half.reshape(-1), p.rho_out)
    L.add_ns_pressure(rest.reshape(-1), p.rho_out)
    return L


@pytest.mark.parametrize("collision", ["bgk", "porous"])
@pytest.mark.parametrize("nx", ODD)
@pytest.mark.parametrize("prec", ["f16", "bf16", "f16q"])
def test_16_bit_odd_rows_equal_the_list_path(nx, collision, prec):
    p = problem(nx, collision)
    a, b = lattice.from_problem(p, prec), list_path(p, prec)
    assert a.launches_per_step() == (1 if nx > 16 else 6) and b.launches_per_step() > 1
    for steps in (1, 2, 40):
        a.step(steps)
        b.step(steps)
        got, ref = a.get_state(), b.get_state()
        for k in ("f", "g", "phi", "q"):
            assert np.array_equal(got[k], ref[k]), (k, steps)
    a.close()
    b.close()


def test_odd_rows_stay_refused():
    """Batches and the step monitor take even rows only, fused planes or not."""
    L = lattice.from_problem(problem(33), "f32")
    with pytest.raises(FmError):
        lattice.Batch([L])
    L.set_monitor(1)
    with pytest.raises(FmError):
        L.step(1)
    L.close()
