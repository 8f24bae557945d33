"""fm_get_fields writes page-locked buffers from one kernel (k_fields) up to
kFieldsDirectBytes a plane, and leaves the stepped representation of the x = 0
plane alone: the same values as the copies into ordinary memory, on both sides
of the size line, in every form and output type, between steps and after the
populations were read back."""
import numpy as np
import pytest
import torch

from fluidmaxxer_b200 import lattice, problems

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "ux", "uy", "uz", "phi", "q")


def pinned(n, dtype):
    return torch.empty(n, dtype=torch.float64 if dtype == np.float64 else torch.float32, pin_memory=True).numpy()


@pytest.mark.parametrize("size", [(16, 6, 5), (33, 9, 7), (64, 32, 32), (128, 128, 64), (130, 128, 64)], ids=str)
@pytest.mark.parametrize("prec", ["f32", "f64", "f16", "f16q"])
def test_equal_to_copies(prec, size):
    p = problems.channel_small(5, *size)
    L, M = lattice.from_problem(p, prec), lattice.from_problem(p, prec)
    for dtype in (np.float32, np.float64):
        out = {k: pinned(L.n, dtype) for k in FIELDS}
        for steps in (1, 6):
            L.step(steps)
            M.step(steps)
            got, ref = L.fields(out=out, dtype=dtype), M.fields(dtype=dtype)
            for k in FIELDS:
                assert np.array_equal(got[k], ref[k]), (k, dtype)
            assert np.array_equal(got["ux"], L.field("ux", dtype=dtype))
    a, b = L.get_state(), M.get_state()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    got, ref = L.fields(out=out, dtype=np.float64), M.fields()   # the plain representation
    for k in FIELDS:
        assert np.array_equal(got[k], ref[k]), k
    L.close()
    M.close()


def test_part_pinned_buffers_take_the_copies():
    p = problems.channel_small(5, 48, 10, 9)
    L = lattice.from_problem(p, "f32")
    L.step(4)
    out = {k: (pinned(L.n, np.float32) if k != "phi" else np.empty(L.n, np.float32)) for k in FIELDS}
    got, ref = L.fields(out=out, dtype=np.float32), L.fields(dtype=np.float32)
    for k in FIELDS:
        assert np.array_equal(got[k], ref[k]), k
    L.close()


def test_overlapping_buffers_keep_the_last_field():
    import ctypes as C

    p = problems.channel_small(5, 48, 10, 9)
    L = lattice.from_problem(p, "f32")
    L.step(30)
    one = pinned(L.n, np.float32)
    ptrs = (C.c_void_p * 6)(*[one.ctypes.data] * 6)
    assert L._lib.fm_get_fields_f32(L.h, ptrs, L.n) == 0
    assert np.array_equal(one, L.field("q", dtype=np.float32))
    L.close()


def test_pair_layout_fields():
    p = problems.channel_small(5, 64, 16, 16)
    L, M = lattice.from_problem(p, "f16"), lattice.from_problem(p, "f16")
    L.set_pair_layout(True)
    out = {k: pinned(L.n, np.float32) for k in FIELDS}
    for steps in (3, 8):
        L.step(steps)
        M.step(steps)
        assert L.storage_layout() == "pair"
        got, ref = L.fields(out=out, dtype=np.float32), M.fields(dtype=np.float32)
        for k in FIELDS:
            assert np.array_equal(got[k], ref[k]), k
    L.close()
    M.close()
