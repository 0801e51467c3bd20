"""A kernel that gives up a wait ends, but not ahead of copies that it has asked for: they would land in the shared memory of whatever block comes next.  Every barrier on which a
tcgen05 kernel announces bytes is drained (tc_drain, csrc/tc_common.cuh) by the thread that announced them.  Read from the sources: no GPU."""
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
            if "tcgen05.alloc" in part and "tc_tma_2d" in part:
                yield f + ":" + re.search(r"(\w+)\s*\(\s*const", part).group(1), part


KERNELS = list(kernels())


def test_there_are_such_kernels():
    assert len(KERNELS) >= 8


@pytest.mark.parametrize("name,text", KERNELS, ids=[n for n, _ in KERNELS])
def test_every_announced_copy_is_waited_for(name, text):
    announced = set(re.findall(r"tc_mbar_expect_tx\(&(\w+)", text))
    if "tc_mbar_expect_tx(bar," in text:             # a loader that is told its barrier
        announced |= set(re.findall(r"load\([^;]*&(\w+)\);", text))
    assert announced
    drained = set(re.findall(r"tc_drain\(&?(\w+)", text))
    assert announced <= drained
