"""Tensor memory of kernels that may start before a grid that is not the library's own has
ended: taken only once they have waited for it, and before they let the next launch start.  Held
earlier, it could keep a grid ahead that allocates late from ever ending.  Read from the
sources: a run that breaks the rule would hang."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vapoursynth-descalemvc_gb300", "csrc")


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernel(name):
    """The kernel's body: from its signature to the closing brace in column 0."""
    text = code(name)
    text = text[text.index("__global__"):]
    return text[:text.index("\n}\n")]


def test_only_the_ring_kernels_allocate():
    assert [f for f in sorted(os.listdir(CSRC)) if "tcgen05.alloc" in code(f)] == ["tring_impl.cuh"]
    assert code("tring_impl.cuh").count("tcgen05.alloc") == 1


@pytest.mark.parametrize("name", ["tring_impl.cuh", "xring_impl.cuh"])
def test_late_allocation_follows_the_wait(name):
    body = kernel(name)
    assert "tcgen05.alloc" not in body
    wait, following = body.index("ring_launch_wait()"), body.index("ring_launch_next()")
    at = [m.start() for m in re.finditer(r"ring_allocate<", body)]
    early, late = at
    assert body[:early].rstrip().endswith("if (!late)")
    assert re.search(r"if \(late\) \{\s*$", body[:late])
    assert early < wait < late < following
