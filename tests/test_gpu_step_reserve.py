"""A step call that cannot have the memory of its outputs fails before its first
step.  The failing allocation is made on the host: memory cannot be had on a
stream under capture, and a call whose samples or monitor rows outgrow what the
lattice holds asks for some."""
import numpy as np
import pytest

from fluidmaxxer_b200 import lattice, problems
from fluidmaxxer_b200._abi import FmError

pytestmark = pytest.mark.gpu

SERIES = 1024   # samples a new series holds; a monitor holds 64 rows


@pytest.mark.parametrize("what", ["series", "monitor"])
def test_failing_call_leaves_the_lattice(what):
    import torch
    from cuda.bindings import runtime as rt

    p = problems.channel_small(5, 32, 16, 16)
    p.sample_every = 1 if what == "series" else 0
    stream = torch.cuda.Stream()
    L, ref = lattice.from_problem(p, "f32", stream=stream.cuda_stream), lattice.from_problem(p, "f32")
    for M in (L, ref):
        if what == "monitor":
            M.set_monitor(7)
        M.step(30)
    L.synchronize()
    mode = rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal
    assert int(rt.cudaStreamBeginCapture(stream.cuda_stream, mode)[0]) == 0
    with pytest.raises(FmError):
        L.step(SERIES)
    rt.cudaStreamEndCapture(stream.cuda_stream)   # the failed request ended it
    rt.cudaGetLastError()
    assert L.step_count == 30
    for steps in (1, 40, SERIES):
        for M in (L, ref):
            M.step(steps)
        got, want = L.fields(), ref.fields()
        for k in got:
            assert np.array_equal(got[k], want[k]), (k, steps)
    if what == "series":
        assert np.allclose(L.breakthrough(), ref.breakthrough(), rtol=1e-12, atol=0.0)   # FP64 sum order
    else:
        got, want = L.monitor(), ref.monitor()
        for k in got:
            assert np.array_equal(got[k], want[k]), k
    L.close()
    ref.close()
