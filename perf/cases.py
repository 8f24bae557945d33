"""Performance cases of the coupled flow + transport + adsorption framework.

Every case is work a user's program has the framework do through its public
Python entry points (``lattice.from_problem``, ``CoupledLattice.step`` /
``fields`` / ``outlet_stats`` / ``breakthrough``, ``Batch.step``,
``adjoint.breakthrough_loss``).  There are four kinds:

* ``flow``    -- advance a lattice by ``steps`` and read the six macroscopic
  fields and the outlet statistics into buffers the program keeps;
* ``job``     -- a whole run: create and set up the lattice, advance it, read
  the fields and the breakthrough series, free it (one point of a sweep);
* ``batch``   -- advance many uneven samples together and read C and q of each;
* ``fit``     -- one iteration of a parameter fit: loss of the breakthrough
  curve and its gradients with respect to the isotherm and the solid fraction.

Three geometries: ``pack`` (random non-overlapping spheres, radius 6),
``grains`` (independent random solid voxels) and ``porous`` (a smooth solid
fraction for the porous collision), made and parametrised as the workloads of
``fluidmaxxer_b200.problems`` are.

``exact`` evaluates the same model on the same inputs in 64 bits, in plain torch.
"""
import dataclasses
import math
import random

import numpy as np
import torch

from fluidmaxxer_b200 import adjoint, lattice, problems, synth

SAMPLE_EVERY = 20          # outlet sampling period of every workload
FIELDS = ("rho", "ux", "uy", "uz", "phi", "q")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    def flow(name, geometry, nx, ny, nz, steps, precision, kind="flow"):
        return dict(name=name, kind=kind, geometry=geometry, nx=nx, ny=ny, nz=nz, steps=steps, precision=precision)

    return [
        # the smallest interactive call: one sampling period of a tiny channel
        flow("channel_32_f32", "grains", 32, 16, 16, 20, "f32"),
        # the small channel workload, ten sampling periods between two outputs
        flow("channel_64_f32", "grains", 64, 32, 32, 200, "f32"),
        # a scanned sample cropped to odd edges: boundary planes not aligned with warps
        flow("grains_odd_f32", "grains", 125, 83, 71, 100, "f32"),
        # the porous-collision workload, forward only
        flow("porous_128_f32", "porous", 128, 64, 64, 200, "f32"),
        # the precision study's crop: the 64-bit reference run ...
        flow("crop_128_f64", "pack", 128, 128, 128, 100, "f64"),
        # ... and the 16-bit form that meets its accuracy bar
        flow("crop_128_f16q", "pack", 128, 128, 128, 100, "f16q"),
        # a mid-sized pack in the other 16-bit format
        flow("pack_256_bf16", "pack", 256, 128, 128, 100, "bf16"),
        # the full-size sphere pack, the headline workload
        flow("pack_512_f32", "pack", 512, 256, 256, 100, "f32"),
        flow("pack_512_f16", "pack", 512, 256, 256, 100, "f16"),
        # uneven samples of a screening study advanced together
        dict(name="batch_16_f32", kind="batch", count=16, steps=60, precision="f32"),
        # one iteration of fitting isotherm and solid fraction to a measured curve
        dict(name="fit_48_f32", kind="fit", nx=48, ny=80, nz=80, steps=240, checkpoint=100, precision="f32"),
        # one run of a parameter sweep, from set-up to results
        flow("job_160_f32", "pack", 160, 96, 96, 200, "f32", kind="job"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choices(("flow", "job", "batch", "fit"), (70, 10, 10, 10))[0]
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 16), steps=20 * rng.randint(1, 3),
                    precision=rng.choice(("f32", "f32", "f16q")))
    if kind == "fit":
        # short beds and enough steps for the flow to reach the outlet: before
        # that the curve does not depend on the solid fraction
        nx = 2 * rng.randint(12, 26)
        return dict(kind=kind, nx=nx, ny=_log_int(rng, 24, 80), nz=_log_int(rng, 24, 80),
                    steps=SAMPLE_EVERY * -(-5 * nx // SAMPLE_EVERY), checkpoint=rng.choice((20, 50, 100)),
                    precision=rng.choice(("f32", "f32", "f64")))
    geometry = rng.choice(("pack", "pack", "grains", "porous"))
    precision = rng.choices(("f32", "f64", "f16", "bf16", "f16q"), (45, 15, 13, 12, 15))[0]
    nx = _log_int(rng, 32, 512)
    if nx % 2 and rng.random() < 0.5:   # even rows are the more common
        nx += 1
    most = (128, 96) if kind == "job" or geometry == "porous" else (256, 256)
    return dict(kind=kind, geometry=geometry, nx=nx, ny=_log_int(rng, 16, most[0]), nz=_log_int(rng, 16, most[1]),
                steps=SAMPLE_EVERY * rng.randint(1, 5 if precision == "f64" else 10) if nx < 256 else
                SAMPLE_EVERY * rng.randint(1, 2 if precision == "f64" else 4),
                precision=precision)


def _batch_sizes(case):
    """The samples' sizes: per-axis edges between 96 and 160, the same for every seed."""
    r = random.Random(1237 + case["count"])
    return [tuple(r.choice((96, 112, 128, 144, 160)) for _ in range(3)) for _ in range(case["count"])]


def work(case):
    """One coupled update reads and writes 26 populations, the concentration's
    previous value (read) and new value (written) stand in the loading's two
    transfers: 19 + 7 populations and q, once in and once out per cell and
    step; about 400 operations.  Reading the fields writes six values a cell."""
    elt = {"f32": 4, "f64": 8}.get(case["precision"], 2)
    per_cell = 52 * elt + (8 if case["precision"] == "f32" else 16)
    if case["kind"] == "batch":
        n = sum(x * y * z for x, y, z in _batch_sizes(case))
        read = 2 * n
    else:
        n = case["nx"] * case["ny"] * case["nz"]
        read = 6 * n
    steps = case["steps"]
    if case["kind"] == "fit":
        # forward, then per backward step the state (read), the adjoint state
        # (read and written) and the solid fraction's gradient
        back = (28 + 2 * 28) * elt + 16
        return {"bytes": float(n * steps * (per_cell + back)), "flops": float(n * steps * 1600)}
    return {"bytes": float(n * steps * per_cell + read * (8 if case["precision"] == "f64" else 4)),
            "flops": float(n * steps * 400)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _problem(geometry, nx, ny, nz, seed, **more):
    if geometry == "grains":
        p = problems.channel_small(seed, nx, ny, nz)
    elif geometry == "pack":
        p = problems.sphere_pack(seed, nx, ny, nz)
    else:
        p = problems.smooth_porous(seed, nx, ny, nz)
        # values that both float types hold
        p.notes["n_s"] = p.notes["n_s"].reshape(-1).astype(np.float32).astype(np.float64)
        p.porosity, p.region = 1.0 - p.notes["n_s"], (p.notes["n_s"] > 0.5).astype(np.uint8)
    return dataclasses.replace(p, **more)


def _problems(case, seed):
    if case["kind"] == "batch":
        r, out = random.Random(int(seed)), []
        for i, (nx, ny, nz) in enumerate(_batch_sizes(case)):
            log = lambda lo, hi: math.exp(r.uniform(math.log(lo), math.log(hi)))  # noqa: E731
            solid = synth.bernoulli(nx, ny, nz, r.uniform(0.5, 0.7), int(seed) * 1000 + i, fluid_lo=4, fluid_hi=4,
                                    walls=True)
            out.append(problems.Problem(nx=nx, ny=ny, nz=nz, solid=solid, tau=0.7, tau_ad=0.6, u_in=(0.01, 0.0, 0.0),
                                        isotherm="langmuir", q_max=log(1, 10), b_langmuir=log(0.1, 5),
                                        k_ldf=log(0.005, 0.1)))
        return out
    if case["kind"] == "fit":
        # a bed that starts filled with carrier at half the feed concentration,
        # so the outlet responds from the first sample on
        return [_problem("porous", case["nx"], case["ny"], case["nz"], int(seed), phi0=0.5, steps=case["steps"])]
    return [_problem(case["geometry"], case["nx"], case["ny"], case["nz"], int(seed))]


def _pinned(n, dtype):
    return torch.empty(n, dtype=torch.float64 if dtype == np.float64 else torch.float32,
                       pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    """The problems, the lattices (or what a job makes them from), and the page-locked buffers results are read into."""
    ps = _problems(case, seed)
    dtype = np.float64 if case["precision"] == "f64" else np.float32
    s = dict(case=case, problems=ps, dtype=dtype)
    if case["kind"] == "batch":
        s["lattices"] = [lattice.from_problem(p, case["precision"]) for p in ps]
        s["batch"] = lattice.Batch(s["lattices"])
        s["out"] = [{k: _pinned(p.n_cells, dtype) for k in ("C", "q")} for p in ps]
    elif case["kind"] == "fit":
        p = ps[0]
        s["lattice"] = lattice.from_problem(p, case["precision"])
        real = torch.float64 if case["precision"] == "f64" else torch.float32
        s["params"] = torch.tensor([p.q_max, p.b_langmuir, p.k_ldf], dtype=real, device=_device())
        s["n_s"] = torch.tensor(p.notes["n_s"], dtype=real, device=_device())
        s["target"] = _target(case)
    else:
        if case["kind"] == "flow":
            s["lattice"] = lattice.from_problem(ps[0], case["precision"])
        s["out"] = {k: _pinned(ps[0].n_cells, dtype) for k in FIELDS}
    return s


def _target(case):
    """A measured curve, sampled every SAMPLE_EVERY steps."""
    m = case["steps"] // SAMPLE_EVERY
    return 0.3 + 0.2 * np.arange(1, m + 1) / m


def run(state):
    case = state["case"]
    if case["kind"] == "flow":
        L = state["lattice"]
        L.step(case["steps"])
        res = dict(L.fields(out=state["out"], dtype=state["dtype"]))
        res["outlet"] = np.array(L.outlet_stats())
        return res
    if case["kind"] == "job":
        with lattice.from_problem(state["problems"][0], case["precision"]) as L:
            L.step(case["steps"])
            res = dict(L.fields(out=state["out"], dtype=state["dtype"]))
            res["breakthrough"] = L.breakthrough()
        return res
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        return [{k: L.field(k, out=o[k], dtype=state["dtype"]) for k in ("C", "q")}
                for L, o in zip(state["lattices"], state["out"])]
    params = state["params"].detach().requires_grad_(True)
    n_s = state["n_s"].detach().requires_grad_(True)
    loss = adjoint.breakthrough_loss(params, n_s, state["problems"][0], state["target"], lattice=state["lattice"],
                                     nsteps=case["steps"], checkpoint_every=case["checkpoint"])
    loss.backward()
    return {"loss": loss.detach(), "params": params.grad, "n_s": n_s.grad}


# ---------------------------------------------------------------------------
# the model in 64 bits
# ---------------------------------------------------------------------------

# velocities and weights of the two lattices; OPP: the opposite direction
C19 = ((0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
       (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1),
       (0, -1, -1))
W19 = (1 / 3,) + (1 / 18,) * 6 + (1 / 36,) * 12
OPP = tuple(C19.index((-x, -y, -z)) for x, y, z in C19)
C7 = C19[:7]
W7 = (1 / 4,) + (1 / 8,) * 6


def _with_column(t, i, column):
    """`t` with its x-column i (0 or -1) replaced."""
    column = column[..., None]
    return torch.cat((column, t[..., 1:]) if i == 0 else (t[..., :-1], column), -1)


class _Model:
    """The coupled step on lists of [nz, ny, nx] planes: D3Q19 pull with half-way
    bounce-back (or porous collision), non-equilibrium velocity inlet, pressure
    outlet, D3Q7 transport with the loading's linear driving force.  Periodic in
    y and z.  Every operation makes new tensors, so it can be differentiated."""

    def __init__(self, p):
        dev, shape = _device(), (p.nz, p.ny, p.nx)
        self.p = p
        t = lambda a: torch.as_tensor(a, device=dev).reshape(shape)  # noqa: E731
        self.porous = p.collision == "porous"
        solid, region = t(p.solid).bool(), p.solid if p.region is None else p.region
        self.solid, self.region = solid, t(region).bool()
        self.porosity = t(np.asarray(p.porosity, np.float64)) if self.porous else None
        self.iso = (p.k_henry, 0.0, p.k_a) if p.isotherm == "linear" else (p.q_max, p.b_langmuir, p.k_ldf)
        self.bounce = []
        for c in C19:
            src = torch.roll(solid, (c[2], c[1], c[0]), (0, 1, 2))
            if c[0]:
                src[..., 0 if c[0] > 0 else -1] = False   # outside the domain: no link
            self.bounce.append(solid | src)
        full = lambda v: torch.full(shape, v, dtype=torch.float64, device=dev)  # noqa: E731
        self.start = ([full(w * p.rho0) for w in W19], [full(w * p.phi0) for w in W7], full(0.0), full(0.0))

    @staticmethod
    def pull(f, c):
        s = torch.roll(f, (c[2], c[1], c[0]), (0, 1, 2))
        if c[0]:
            i = 0 if c[0] > 0 else -1
            s = _with_column(s, i, f[..., i])
        return s

    @staticmethod
    def moments(f):
        rho, j = f[0], [0.0, 0.0, 0.0]
        for k in range(1, 19):
            rho = rho + f[k]
            for a in range(3):
                if C19[k][a]:
                    j[a] = j[a] + C19[k][a] * f[k]
        return rho, [a / rho for a in j]

    @staticmethod
    def feq(k, rho, u, u2):
        c = C19[k]
        e = sum(c[a] * u[a] for a in range(3) if c[a]) if k else 0.0
        return W19[k] * rho * (1.0 + 3.0 * e + 4.5 * e * e - 1.5 * u2)

    def step(self, f, g, phi, q, iso=None, porosity=None):
        p = self.p
        iso = self.iso if iso is None else iso
        # velocity inlet from the x = 1 cells
        near = [a[..., 1] for a in f]
        rho, u = self.moments(near)
        u2, b2 = sum(a * a for a in u), sum(a * a for a in p.u_in)
        f = [_with_column(f[k], 0, self.feq(k, rho, p.u_in, b2) + near[k] - self.feq(k, rho, u, u2))
             for k in range(19)]
        # pull and collide
        s = [self.pull(f[k], C19[k]) for k in range(19)]
        if not self.porous:
            s = [torch.where(self.bounce[k], f[OPP[k]], s[k]) for k in range(19)]
        del f
        rho, u = self.moments(s)
        if self.porous:
            por = (self.porosity if porosity is None else porosity).clamp(0.0, 1.0)
            u = [a * por for a in u]
        u2 = sum(a * a for a in u)
        omega = 1.0 / max(p.tau, 0.5001)
        for k in range(19):
            n = s[k] + omega * (self.feq(k, rho, u, u2) - s[k])
            s[k] = n if self.porous else torch.where(self.solid, s[k], n)
        # pressure outlet from the x = nx - 2 cells
        u = [a[..., -2] for a in self.moments([a[..., -2:] for a in s])[1]]
        u2 = sum(a * a for a in u)
        f = [_with_column(s[k], -1, self.feq(k, p.rho_out, u, u2) + 0.0 * u2) for k in range(19)]
        u = self.moments(f)[1]
        # adsorption: linear driving force from the previous concentration
        ce = phi.clamp(min=p.min_conc) - p.min_conc
        qeq = iso[0] * ce if p.isotherm == "linear" else iso[0] * (iso[1] * ce / (1.0 + iso[1] * ce))
        dq = torch.where(self.region, iso[2] * (qeq - q), 0.0)
        # transport
        s = [self.pull(g[k], C7[k]) for k in range(7)]
        phi = sum(s[1:], s[0]).clamp(min=p.min_conc)
        om = 1.0 / p.tau_ad
        g = []
        for k in range(7):
            a = [i for i in range(3) if C7[k][i]]
            geq = W7[k] * phi * (1.0 + 4.0 * C7[k][a[0]] * u[a[0]]) if a else W7[k] * phi
            n = s[k] + om * (geq - s[k]) - W7[k] * dq
            n = _with_column(n, 0, torch.full_like(n[..., 0], p.c_in * W7[k]))
            g.append(_with_column(n, -1, n[..., -2]))
        return f, g, phi, q + dq

    def advance(self, steps):
        x, series = self.start, [float(self.start[2][..., -1].mean())]
        self.start = None
        with torch.no_grad():
            for i in range(steps):
                x = self.step(*x)
                if (i + 1) % SAMPLE_EVERY == 0:
                    series.append(float(x[2][..., -1].mean()))
        return x, np.array(series)

    def fields(self, x):
        rho, u = self.moments(x[0])
        flat = lambda t: t.reshape(-1).cpu()  # noqa: E731
        return dict(zip(FIELDS, map(flat, (rho, *u, x[2], x[3]))))


def _exact_fit(case, p):
    """Reverse mode over the stored states, one differentiated step at a time."""
    m = _Model(p)
    states, target = [m.start], _target(case)
    with torch.no_grad():
        for _ in range(case["steps"]):
            states.append(m.step(*states[-1]))
    dev = _device()
    iso = torch.tensor(m.iso, dtype=torch.float64, device=dev, requires_grad=True)
    por = m.porosity.clone().requires_grad_(True)
    zero = lambda: torch.zeros(m.solid.shape, dtype=torch.float64, device=dev)  # noqa: E731
    lam = [zero() for _ in range(28)]
    g_iso, g_por, loss = torch.zeros(3, dtype=torch.float64, device=dev), zero(), 0.0
    rows = p.ny * p.nz
    for t in range(case["steps"], 0, -1):
        if t % SAMPLE_EVERY == 0:
            r = float(states[t][2][..., -1].mean()) - target[t // SAMPLE_EVERY - 1]
            loss += r * r
            lam[26] = lam[26].clone()
            lam[26][..., -1] += 2.0 * r / rows
        states.pop()
        f, g, phi, q = states[t - 1]
        x = [a.detach().requires_grad_(True) for a in (*f, *g, phi, q)]
        y = m.step(x[:19], x[19:26], x[26], x[27], iso, por)
        got = torch.autograd.grad((*y[0], *y[1], y[2], y[3]), [*x, iso, por], lam, allow_unused=True)
        lam = [zero() if a is None else a for a in got[:28]]
        g_iso += got[28]
        g_por += got[29]
    return {"loss": torch.tensor(loss, dtype=torch.float64), "params": g_iso, "n_s": -g_por.reshape(-1)}


def exact(case, seed):
    ps = _problems(case, seed)
    if case["kind"] == "fit":
        return _exact_fit(case, ps[0])
    if case["kind"] == "batch":
        out = []
        for p in ps:
            x, _ = _Model(p).advance(case["steps"])
            out.append({"C": x[2].reshape(-1).cpu(), "q": x[3].reshape(-1).cpu()})
        return out
    m = _Model(ps[0])
    x, series = m.advance(case["steps"])
    res = m.fields(x)
    if case["kind"] == "flow":
        c = x[2][..., -1]
        # ahead of the front the outlet holds less than one step of the 16-bit formats
        res["outlet"] = (np.array([float(c.mean()), float(c.min()), float(c.max())])
                         if case["precision"] in ("f32", "f64") else None)
    else:
        res["breakthrough"] = series if case["precision"] in ("f32", "f64") else None
    return res
