"""Device initialisation is ordered with the streams that use it.

A cudaMemset or cudaMemcpy on the legacy default stream is not waited for by
non-blocking streams (the serving engine's workers, PyTorch's side streams):
work counters zeroed that way were still garbage, or were zeroed in mid-run,
when a worker's first kernel on a grid read them.  Only grid creation uses the
legacy stream, and it waits for it before it hands the grid out.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pisces-1_gb300", "csrc")


def test_only_grid_creation_uses_the_legacy_stream():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".cpp")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        calls = re.findall(r"\bcuda(?:Memset|Memcpy)\s*\(", text)
        assert not calls or name == "pg_grid.cu", (name, calls)


def test_grid_creation_waits_for_the_legacy_stream():
    with open(os.path.join(CSRC, "pg_slice.cu")) as f:
        text = f.read()
    body = text[text.index("pg_status slice_grid("):]
    body = body[:body.index("\n}\n")]
    assert "cudaStreamSynchronize(0)" in body  # the last step of pg_grid_create
    with open(os.path.join(CSRC, "pg_grid.cu")) as f:
        text = f.read()
    tail = text[text.index("pg::slice_grid(g)"):text.index('extern "C" pg_status pg_grid_destroy')]
    assert "cudaMem" not in tail
