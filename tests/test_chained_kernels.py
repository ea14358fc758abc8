"""Launches that overlap (``launch_chained``): where they are used."""
import glob
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "afid-murphfi_b200", "csrc")
SOURCES = {os.path.basename(p): open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def test_a_batch_runs_and_is_tuned_with_plain_launches():
    # its steps are captured, where programmatic edges cost more than plain ones
    src = SOURCES["afid_batch.cu"]
    assert "launch_chained(" not in src and "chain_begin()" not in src
    # switched off once, at creation and thus before the autotuner, and never on again
    assert src.count("L.chained") == 1 and "b->ctx->L.chained = false;" in src
    assert src.index("b->ctx->L.chained = false;") < src.index("int afid_batch_step(")
