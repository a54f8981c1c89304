"""CPU: properties of the kernel sources that no run can be relied on to show.

A statement that copies to shared memory, waits or synchronises orders the
plain loads and stores around it only if the compiler is told so: without a
"memory" clobber it may move them across.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu_msm_b200", "csrc")
ORDERING = re.compile(r'asm\s+volatile\s*\(\s*"(cp\.async|bar\.|barrier\.|mbarrier\.|griddepcontrol\.|fence\.|membar)')


def ordering_statements():
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        if not path.endswith((".cu", ".cuh", ".h")):
            continue
        src = open(path).read()
        for m in ORDERING.finditer(src):
            yield os.path.basename(path), src.count("\n", 0, m.start()) + 1, src[m.start():src.index(");", m.start())]


def test_there_are_ordering_statements():
    assert len(list(ordering_statements())) >= 8


@pytest.mark.parametrize("where,line,text", list(ordering_statements()), ids=lambda v: str(v)[:40])
def test_ordering_statements_clobber_memory(where, line, text):
    assert '"memory"' in text, (where, line, text)
