"""Odd row lengths at the sizes where the direct-planes step changes its launch:
several resident waves, with the flag words fetched ahead; beyond 2.2M cells,
blocks of 256 threads and the next step's blocks placed while this one still
stores; and a 16-bit lattice whose pulls need unsigned offsets.  Boundary cells
and their neighbours fall into different warps and blocks throughout."""
import dataclasses

import numpy as np
import pytest

from fluidmaxxer_b200 import lattice, problems, slabs, synth
from fluidmaxxer_b200._abi import check
from oracle.oracle import Oracle

from .test_gpu_direct_planes import list_path

pytestmark = pytest.mark.gpu

SIZES = [(125, 45, 37), (157, 125, 121)]   # 208k and 2.4M cells
CALLS = (1, 4, 3)                          # steps: chained ones in the later calls


def problem(nx, ny, nz):
    solid = synth.bernoulli(nx, ny, nz, 0.3, 2000 + nx, fluid_lo=0, fluid_hi=0, walls=True)
    solid = solid.reshape(nz, ny, nx)
    solid[9:14, 9:14, 20:60] = 1           # whole sectors at rest
    return problems.Problem(nx=nx, ny=ny, nz=nz, solid=solid.reshape(-1), tau=0.7, tau_ad=0.6, u_in=(0.02, 0.0, 0.0),
                            isotherm="langmuir", q_max=3.0, b_langmuir=1.2, k_ldf=0.05)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_bit_exact_vs_oracle(size, prec):
    p = problem(*size)
    L = lattice.from_problem(p, prec)
    o = Oracle(p, "restated", prec)
    assert L.launches_per_step() == 1
    for steps in CALLS:
        L.step(steps)
        o.step(steps)
        got, ref = L.get_state(), o.get(populations=True)
        for k in ("f", "g", "phi", "q"):
            assert np.array_equal(got[k], ref[k]), (k, steps)
    L.close()
    o.close()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("prec", ["f16", "bf16", "f16q"])
def test_16_bit_equals_the_list_path(size, prec):
    p = problem(*size)
    a, b = lattice.from_problem(p, prec), list_path(p, prec)
    assert a.launches_per_step() == 1 and b.launches_per_step() > 1
    for steps in CALLS:
        a.step(steps)
        b.step(steps)
        got, ref = a.get_state(), b.get_state()
        for k in ("f", "g", "phi", "q"):
            assert np.array_equal(got[k], ref[k]), (k, steps)
    a.close()
    b.close()


def test_unsigned_offsets_step_as_the_tile():
    """A lattice periodic in z whose geometry repeats every 8 planes advances as
    its 8-plane tile does (test_gpu_large), here with rows of 511 cells: 121M
    cells, past the signed offsets' range."""
    import torch

    nx, ny, tile, nz = 511, 512, 8, 464
    solid = (np.random.default_rng(7).random((tile, ny, nx)) < 0.15).astype(np.uint8)
    solid[:, :, :3] = 0
    solid[:, :, nx - 3:] = 0
    p = problems.Problem(nx=nx, ny=ny, nz=tile, solid=solid.reshape(-1), periodic=(False, True, True),
                         isotherm="linear", sample_every=0, steps=6)

    def planes(L, zs):
        out = []
        for z in zs:
            t = torch.empty(slabs.PLANE_POPULATIONS * nx * ny * slabs.ELEMENT_BYTES["f16"], dtype=torch.uint8,
                            device="cuda")
            check(L._lib.fm_pack_zplane(L.h, int(z), t.data_ptr()))
            out.append(t)
        torch.cuda.synchronize()
        return out

    small = lattice.from_problem(p, "f16", probe=False)
    small.step(6)
    ref = planes(small, range(tile))
    small.close()
    big = lattice.from_problem(dataclasses.replace(p, nz=nz, solid=np.tile(solid, (nz // tile, 1, 1)).reshape(-1)),
                               "f16", probe=False)
    assert big.step_kernel() == "one-cell-wide" and big.launches_per_step() == 1
    big.step(6)
    zs = [0, 1, tile - 1, tile, nz // 2, nz // 2 + 1, nz - tile, nz - 2, nz - 1]
    got = planes(big, zs)
    big.close()
    lattice.trim_memory()
    torch.cuda.empty_cache()
    for z, g in zip(zs, got):
        assert torch.equal(g, ref[z % tile]), z
