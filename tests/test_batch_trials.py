"""Batch.autotune compares the launch modes by trial steps.  Mode 3 writes the
x = 0 side plane and every cell's C only on steps whose outputs may be read, so
its trials have to ask for the outputs a run of steps asks for; which outputs
a trial asked for cannot be seen from its results, which are taken back, so the
source is held to the rule."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def body(text, head):
    start = text.index(head)
    return text[start:text.index("\n}\n", start)]


def test_trials_ask_for_the_outputs_of_a_run():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "fluidmaxxer_b200", "csrc", "fm_abi.cu")).read())
    for head in ("int batch_one(fm_batch* B, long long", "int fm_batch_autotune(fm_batch* B, int"):
        calls = re.findall(r"batch_dispatch_step\((.*)\);", body(text, head))
        assert calls and all("batch_outputs(B, s" in c for c in calls), (head, calls)
    rule = body(text, "int batch_outputs(const fm_batch* B, long long")
    assert "last ? fm::kOutX0" in rule and "last || batch_sampled(B, s) ? fm::kOutC" in rule
