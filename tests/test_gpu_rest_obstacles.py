"""Obstacles at rest keep their populations without being stepped (kRest), and C
is written between outputs in the adsorption region only (kKeepC): geometries
with solid runs longer than a sector of any storage form, and every way an
obstacle can leave the rest state."""
import numpy as np
import pytest

from fluidmaxxer_b200 import lattice, problems
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

KEYS = ("f", "g", "phi", "q")


def problem(nx, seed=3, **more):
    """Solid blocks with edges of 1 to 24 cells, walls, and a region of its own."""
    ny, nz = 12, 10
    r = np.random.default_rng(seed)
    solid = np.zeros((nz, ny, nx), np.uint8)
    for _ in range(14):
        x, y, z = r.integers(0, nx), r.integers(0, ny), r.integers(0, nz)
        solid[z:z + r.integers(1, 5), y:y + r.integers(1, 6), x:x + r.integers(1, 25)] = 1
    solid[0], solid[-1], solid[:, 0], solid[:, -1] = 1, 1, 1, 1
    region = np.zeros((nz, ny, nx), np.uint8)
    region[:, :, nx // 3:nx // 2] = 1
    region |= (r.uniform(size=region.shape) < 0.01).astype(np.uint8)
    args = dict(nx=nx, ny=ny, nz=nz, solid=solid.reshape(-1), region=region.reshape(-1), tau=0.7, tau_ad=0.6,
                u_in=(0.02, 0.0, 0.0), isotherm="langmuir", q_max=3.0, b_langmuir=1.2, k_ldf=0.05, phi0=0.3)
    args.update(more)
    return problems.Problem(**args)


@pytest.mark.parametrize("nx", [16, 33, 61, 64, 90, 128])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_bit_exact_vs_oracle(nx, prec):
    p = problem(nx)
    L = lattice.from_problem(p, prec)
    o = Oracle(p, "restated", prec)
    for steps in (1, 6, 45):
        L.step(steps)
        o.step(steps)
        got, ref = L.get_state(), o.get(populations=True)
        for k in KEYS:
            assert np.array_equal(got[k], ref[k]), (k, steps)
    got, ref = L.breakthrough(), o.get()["c_out"]
    assert np.allclose(got, ref, rtol=1e-12, atol=1e-300)
    L.close()
    o.close()


@pytest.mark.parametrize("more", [{}, dict(isotherm="none"), dict(coupling=False),
                                  dict(ns_inlet="none", ns_outlet="none", ad_inlet="none", ad_outlet="none",
                                       periodic=(True, True, True))], ids=["full", "inert", "uncoupled", "closed"])
@pytest.mark.parametrize("prec", ["f32", "f64", "f16", "bf16", "f16q"])
def test_equals_monitored_steps(prec, more):
    """Monitored steps write every cell on every step."""
    p = problem(96, **more)
    a, b = lattice.from_problem(p, prec), lattice.from_problem(p, prec)
    b.set_monitor(1)
    for steps in (1, 7, 40):
        a.step(steps)
        b.step(steps)
        got, ref = a.get_state(), b.get_state()
        for k in KEYS:
            assert np.array_equal(got[k], ref[k]), (k, steps)
    a.close()
    b.close()


@pytest.mark.parametrize("prec", ["f32", "f16"])
@pytest.mark.parametrize("how", ["state", "mask", "copy", "porous"])
def test_obstacles_set_moving_are_stepped(prec, how):
    """Populations from outside, obstacles placed into flow, the copy benchmark's
    scrambled buffer, and a spell of porous collision: the next steps equal
    those of a lattice that writes every cell."""
    p = problem(96)
    lats = [lattice.from_problem(p, prec) for _ in range(2)]
    lats[1].set_monitor(1)
    r = np.random.default_rng(5)
    state = None
    for L in lats:
        L.step(9)
        if how == "state":
            if state is None:
                state = L.get_state()
                state["f"] *= 1.0 + 0.01 * r.uniform(size=state["f"].shape)
            L.set_state(f=state["f"])
        elif how == "mask":
            solid = p.solid.reshape(p.nz, p.ny, p.nx).copy()
            solid[3:6, 3:9, 30:62] = 1
            L.set_obstacle_mask(solid.reshape(-1))
        elif how == "copy":
            L.bench_pull_copy(2)
        else:
            L.set_collision("porous")
            L.set_porosity(np.full(L.n, 0.6))
            L.step(3)
            L.set_collision("bgk")
        for steps in (1, 2, 11):
            L.step(steps)
    a, b = (L.get_state() for L in lats)
    for k in KEYS:
        assert np.array_equal(a[k], b[k]), k
    # a new start is at rest again
    for L in lats:
        L.init_equilibrium()
        L.step(12)
    a, b = (L.get_state() for L in lats)
    for k in KEYS:
        assert np.array_equal(a[k], b[k]), k
    for L in lats:
        L.close()


def test_batch_reads_every_cell_between_calls():
    p, q = problem(64), problem(48, seed=8)
    lats = [lattice.from_problem(x, "f32") for x in (p, q)]
    with_batch = lattice.Batch(lats)
    alone = [lattice.from_problem(x, "f32") for x in (p, q)]
    for steps in (3, 41, 20):
        with_batch.step(steps)
        for L, A in zip(lats, alone):
            A.step(steps)
            got, ref = L.get_state(), A.get_state()
            for k in KEYS:
                assert np.array_equal(got[k], ref[k]), (k, steps)
    for L, A in zip(lats, alone):
        assert np.allclose(L.breakthrough(), A.breakthrough(), rtol=1e-12, atol=1e-300)
    with_batch.close()
    for L in lats + alone:
        L.close()
