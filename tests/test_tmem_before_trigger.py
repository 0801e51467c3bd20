"""A kernel that allocates TMEM lets its successor start (griddepcontrol.launch_dependents) only behind that allocation: a successor that allocates
too holds its columns until the kernel has completed, so a block that came to its allocation later would wait for ever.  Read from the sources: no GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hip_llama.cpp_b200", "csrc")


def kernels():
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for part in re.split(r"(?=\b__global__\b)", text)[1:]:
            if "tcgen05.alloc" in part:
                yield f + ":" + re.search(r"(\w+)\s*\(\s*const", part).group(1), part


KERNELS = list(kernels())


def test_there_are_such_kernels():
    assert len(KERNELS) >= 6


@pytest.mark.parametrize("name,text", KERNELS, ids=[n for n, _ in KERNELS])
def test_allocated_and_published_ahead_of_the_trigger(name, text):
    alloc = text.index("tcgen05.alloc")
    published = text.index("__syncthreads()", alloc)
    for m in re.finditer(r"\b(pdl_trigger|hyb_pdl_enter)\(\)", text):
        assert m.start() > published
