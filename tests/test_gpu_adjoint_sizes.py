"""k_adj_step at row lengths where its paths change: rows shorter than a warp
(several inlet rows a warp), rows across warps, warps without an x-face, and
cells whose every warp lies on a y/z face.  FP64 gradients against central
differences of the FP64 forward, 1e-6 of the largest component."""
import numpy as np
import pytest

from fluidmaxxer_b200 import lattice, problems, synth

pytestmark = pytest.mark.gpu

STEPS = 40


def problem(nx, ny, nz, collision, periodic):
    n = nx * ny * nz
    r = np.random.default_rng(nx * 7 + ny)
    args = dict(nx=nx, ny=ny, nz=nz, periodic=periodic, tau=0.8, tau_ad=0.7, u_in=(0.02, 0.0, 0.0), phi0=0.4,
                isotherm="langmuir", q_max=2.0, b_langmuir=1.1, k_ldf=0.06, sample_every=10, steps=STEPS,
                region=(r.uniform(size=n) < 0.5).astype(np.uint8))
    if collision == "porous":
        return problems.Problem(solid=np.zeros(n, np.uint8), collision="porous",
                                porosity=r.uniform(0.3, 0.9, n), **args)
    return problems.Problem(solid=synth.bernoulli(nx, ny, nz, 0.25, nx, fluid_lo=0, fluid_hi=0, walls=False), **args)


def loss(p, target, params=None, porosity=None):
    L = lattice.from_problem(p, "f64")
    if params is not None:
        L.set_isotherm_langmuir(p.region, *params)
    if porosity is not None:
        L.set_porosity(porosity)
    L.init_equilibrium()
    L.step(STEPS)
    s = L.breakthrough()[1:]
    L.close()
    return float(np.sum((s - target) ** 2))


@pytest.mark.parametrize("collision", ["bgk", "porous"])
@pytest.mark.parametrize("periodic", [(False, True, True), (False, False, False), (True, True, True)],
                         ids=["yz", "none", "xyz"])
@pytest.mark.parametrize("size", [(4, 6, 5), (14, 5, 4), (34, 4, 3), (66, 5, 5), (130, 2, 6)], ids=str)
def test_gradients_match_differences(size, periodic, collision):
    p = problem(*size, collision, periodic)
    target = np.linspace(0.1, 0.3, STEPS // p.sample_every)
    L = lattice.from_problem(p, "f64")
    _, gp, gpor = L.adjoint_breakthrough(STEPS, target, checkpoint_every=15, max_stored_states=4)
    L.close()
    params = np.array([p.q_max, p.b_langmuir, p.k_ldf])
    for i in range(3):
        h = 1e-5 * params[i]
        up, dn = params.copy(), params.copy()
        up[i] += h
        dn[i] -= h
        fd = (loss(p, target, up) - loss(p, target, dn)) / (2 * h)
        assert abs(fd - gp[i]) <= 1e-6 * np.abs(gp).max(), (i, fd, gp[i])
    if collision == "porous":
        big = np.abs(gpor).max()
        for c in np.argsort(np.abs(gpor))[-3:]:
            up, dn = p.porosity.copy(), p.porosity.copy()
            up[c] += 1e-4
            dn[c] -= 1e-4
            fd = (loss(p, target, porosity=up) - loss(p, target, porosity=dn)) / 2e-4
            assert abs(fd - gpor[c]) <= 1e-6 * big + 1e-13, (c, fd, gpor[c])
