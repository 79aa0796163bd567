"""Rules that the kernels' source keeps, where a break shows on the GPU only now
and then.

Named barriers: bar.sync and bar.arrive count a warp at its first arrival, so a
warp that may have diverged is made whole (__syncwarp) in the statement before
one."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bola_gb300", "csrc")
UNITS = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def source(path):
    """The code without its comments, one statement's whitespace like another's."""
    text = open(path).read()
    text = re.sub(r"//[^\n]*", "", text)
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("path", UNITS, ids=os.path.basename)
def test_warps_are_whole_at_named_barriers(path):
    text = source(path)
    for m in re.finditer(r'asm volatile\("bar\.(sync|arrive)', text):
        before = text[:m.start()].rstrip()
        assert before.endswith("__syncwarp();"), text[max(0, m.start() - 200):m.end() + 40]
