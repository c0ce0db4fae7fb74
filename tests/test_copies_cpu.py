"""Every write to device memory by the host is queued on the stream whose
kernels read it.  The handles' streams are non-blocking: work on the legacy
stream (cudaMemcpy, cudaMemset) is not ordered with theirs, and a copy from
pageable memory may still be on its way when cudaMemcpy returns, so a kernel
launched next could read what was there before.  Checked on the sources: on a
GPU the difference shows by chance only."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gsbn_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")))


def calls(text, name):
    """the argument text of every call of `name` outside comments"""
    text = re.sub(r"/\*.*?\*/", " ", text, flags=re.S)
    for m in re.finditer(r"\b" + name + r"\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        yield text[m.end():k - 1]


@pytest.mark.parametrize("source", SOURCES)
def test_writes_are_queued_on_a_stream(source):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    for name in ("cudaMemset", "cudaMemcpyToSymbol", "cudaMemcpy2D"):
        assert not list(calls(text, name)), name
    for args in calls(text, "cudaMemcpy"):
        assert args.rstrip().endswith("cudaMemcpyDeviceToHost"), args
    for name in ("cudaMemcpyAsync", "cudaMemsetAsync", "cudaMemcpyToSymbolAsync"):
        for args in calls(text, name):
            assert re.search(r"stream\w*\s*$", args), args
