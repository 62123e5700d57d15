"""Every tcgen05 operation of the kernels (MMA issue, TMEM load, TMEM store) that
follows a wait on an mbarrier has a tcgen05.fence::after_thread_sync between
the two: without it the order between the operations whose completion was
waited for and the new one is not given (a TMEM store may then meet the reads
of earlier MMAs).  A missing fence shows in no value reliably, so the sources
are read: from each operation back to the last wait before it.  No GPU."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "superdca_gb300", "csrc")

WAIT = re.compile(r"\bmbar_wait(_warp)?\(")
FENCE = "tcgen05.fence::after_thread_sync"
OP = re.compile(r"\b(mma_f16\w*|tmem_ld\d+|tmem_st\d+)\(")


def _kernels(src):
    """Bodies of the functions that wait (one per top-level brace block)."""
    src = re.sub(r"//[^\n]*", "", src)
    for m in re.finditer(r"^\{\n(.*?)^\}", src, re.M | re.S):
        if WAIT.search(m.group(1)):
            yield m.group(1)


@pytest.mark.parametrize("name,operations", [("kernels_tc.cu", 10), ("mlp.cu", 4)])
def test_fence_between_wait_and_operation(name, operations):
    with open(os.path.join(CSRC, name)) as f:
        src = f.read()
    seen = 0
    for body in _kernels(src):
        for m in OP.finditer(body):
            waits = [w.end() for w in WAIT.finditer(body, 0, m.start())]
            if not waits:
                continue
            seen += 1
            assert FENCE in body[waits[-1]:m.start()], (name, body[max(0, m.start() - 400):m.end()])
    assert seen >= operations, seen
