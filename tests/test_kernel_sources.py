"""CPU: rules of the kernel sources that no run can show to be kept."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparse_b200", "csrc")


def _kernels():
    """(file, name, body) of every `__global__` function."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, name)).read(), flags=re.S)
        for m in re.finditer(r"__global__", text):
            open_brace = text.index("{", m.end())
            depth, end = 1, open_brace + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            head = text[m.end():open_brace]
            yield name, re.findall(r"(\w+_kernel)\s*\(", head)[-1], text[open_brace + 1:end - 1]


DEPENDENT = [(f, k, b) for f, k, b in _kernels() if "pdl_launch_dependents" in b or "pdl_wait" in b]


@pytest.mark.parametrize("body", [b for _, _, b in DEPENDENT], ids=["%s:%s" % (f, k) for f, k, _ in DEPENDENT])
def test_every_thread_waits_for_the_launch_before_it(body):
    """A kernel that may start early waits once, unconditionally, and only declarations,
    index arithmetic and L2 prefetches stand in front of the wait."""
    waits = [m.start() for m in re.finditer(r"pdl_wait\(\)", body)]
    assert len(waits) == 1
    front = body[:waits[0]]
    assert front.count("{") == front.count("}")
    assert front.rstrip().endswith((";", "}"))            # not the branch of an if
    assert not re.search(r"\breturn\b|__ldg|\bld_|\batomic|ld\.global|st\.global", front)
