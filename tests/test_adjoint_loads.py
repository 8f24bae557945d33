"""A backward step of the adjoint may start while the launch before it drains
(programmatic dependent launch), so what that launch writes must not be read
through the read-only path or ahead of the wait.  Which load the compiler
picks cannot be provoked by a run, so the source is held to the rule."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def source():
    text = open(os.path.join(ROOT, "fluidmaxxer_b200", "csrc", "fm_adjoint.cuh")).read()
    return re.sub(r"//[^\n]*", "", text)


def test_inputs_of_a_chained_backward_step_are_not_read_only():
    text = source()
    args = re.search(r"struct AdjArgs \{.*?\n\};", text, re.S).group(0)
    assert "__restrict__" not in args
    kernel = text[text.index("k_adj_step(const AdjArgs"):text.index("k_adj_fold")]
    assert kernel.index("pdl_wait()") < kernel.index("ld_adj(")
    for name in ("A.lfi1", "A.lgi1", "A.lphi1", "A.lq1", "a.phi", "a.q"):
        assert not re.search(re.escape(name) + r"\s*\[", kernel), name
    gathers = text[text.index("gather19_fast(const R*"):text.index("static_assert(cx19(1)")]
    assert not re.search(r"(\bbase|\bl)\s*\[|__restrict__", gathers)
