"""The rule by which fm_get_fields lets a kernel store straight into the caller's
buffers: page-locked ranges the device may write have to cover the whole
buffer.  The rule is checked on made-up ranges without a GPU; a buffer with a
gap is never stored to."""
import numpy as np
import pytest

from fluidmaxxer_b200 import _abi

K = 4096


def span(ranges, p, nbytes, align=4):
    a = np.array([r[0] for r in ranges], np.uint64)
    b = np.array([r[1] for r in ranges], np.uint64)
    w = np.array([r[2] if len(r) > 2 else 1 for r in ranges], np.int32)
    rc = _abi.lib().fm_debug_host_span(a.ctypes.data, b.ctypes.data, w.ctypes.data, len(ranges), p, nbytes, align)
    assert rc in (0, 1)
    return bool(rc)


@pytest.mark.parametrize("ranges, p, nbytes, want", [
    ([(8 * K, 4 * K)], 8 * K, 4 * K, True),                          # the whole range
    ([(8 * K, 4 * K)], 8 * K + 12, K, True),                         # inside it
    ([(8 * K, 4 * K)], 8 * K + 4, 4 * K, False),                     # past its end
    ([(8 * K, 4 * K)], 8 * K - 4, K, False),                         # before its start
    ([(8 * K, K), (10 * K, K)], 8 * K, 3 * K, False),                # both ends locked, a page between them not
    ([(8 * K, K), (9 * K, K), (10 * K, K)], 8 * K, 3 * K, True),     # three registrations side by side
    ([(8 * K, K), (9 * K, K, 0), (10 * K, K)], 8 * K, 3 * K, False), # the middle one read-only
    ([(8 * K, 4 * K, 0)], 8 * K, K, False),                          # read-only
    ([(8 * K, 4 * K)], 8 * K + 2, K, False),                         # not on a value's boundary
    ([], 8 * K, K, False),                                           # ordinary memory
    ([(8 * K, 0)], 8 * K, K, False),                                 # an empty range does not end the walk
], ids=str)
def test_ranges_must_cover_the_buffer(ranges, p, nbytes, want):
    assert span(ranges, p, nbytes) == want


@pytest.mark.gpu
def test_registered_buffers_receive_the_fields():
    """Fields into one registration, and across two side by side."""
    import torch

    from fluidmaxxer_b200 import lattice, problems

    rt = torch.cuda.cudart()
    L = lattice.from_problem(problems.channel_small(5, 64, 16, 16), "f32")
    L.step(7)
    ref = L.fields(dtype=np.float32)
    raw = np.zeros(L.n + 2 * K, np.float32)
    skip = -raw.ctypes.data % K // 4
    page = raw[skip:]
    base, size = page.ctypes.data, L.n * 4   # 16 pages
    for split in (size, size // 2):
        parts = [(base, split)] + ([(base + split, size - split)] if split < size else [])
        for at, nbytes in parts:
            assert int(rt.cudaHostRegister(at, nbytes, 0)) == 0
        try:
            for k in ("rho", "ux", "uy", "uz", "phi", "q"):
                page[:L.n] = np.nan
                pinned = {j: torch.empty(L.n, pin_memory=True).numpy() for j in ref}
                pinned[k] = page[:L.n]
                got = L.fields(out=pinned, dtype=np.float32)
                assert np.array_equal(got[k], ref[k]), (k, split)
        finally:
            for at, _ in parts:
                rt.cudaHostUnregister(at)
    L.close()
