"""Rules that the kernels' source keeps, where a break shows on the GPU only now
and then.

Named barriers: bar.sync and bar.arrive count a warp at its first arrival, so a
warp that may have diverged is made whole (__syncwarp) in the statement before
one.

Programmatic dependents: a kernel that waits for the one before it
(griddepcontrol.wait) has started before that one's results are final, so its
operands are not const __restrict__, which declares them constant during the
whole kernel and allows loads that need not see another kernel's stores.

Function attributes: they belong to a context and are shared by its threads, so
no static of the process remembers that they have been asked for once (PerContext
remembers for which context), and the same shared memory is asked for always (a
size of the call's own would lower another thread's limit)."""
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


def closing(text, at, opening, shutting):
    """Index of the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == opening) - (text[i] == shutting)
        if depth == 0:
            return i
    raise ValueError(text[at:at + 80])


def kernels(text):
    """(name, parameters, body) of every kernel defined in `text`."""
    for m in re.finditer("__global__", text):
        at = m.end()
        while True:  # past __launch_bounds__(...) and the like, to the name's parenthesis
            start = text.index("(", at)
            name = re.search(r"(\w+)\s*$", text[at:start]).group(1)
            end = closing(text, start, "(", ")")
            if not name.startswith("__"):
                break
            at = end + 1
        if text[end + 1:].lstrip().startswith("{"):
            body = text.index("{", end)
            yield name, text[start:end], text[body:closing(text, body, "{", "}")]


@pytest.mark.parametrize("path", UNITS, ids=os.path.basename)
def test_programmatic_dependents_take_plain_pointers(path):
    for name, parameters, body in kernels(source(path)):
        if re.search(r"grid_dependency_wait|griddepcontrol\.wait|\bInParallel\b", body):
            assert not re.search(r"const\s+[\w:]+(\s+\w+)?\s*\*\s*__restrict__", parameters), name


@pytest.mark.parametrize("path", UNITS, ids=os.path.basename)
def test_function_attributes_belong_to_a_context(path):
    text = source(path)
    assert not re.search(r"static (bool|size_t|int) \w*attr\w*", text)
    if os.path.basename(path) == "calibrate.cu":  # (probes, which have the device to themselves)
        return
    for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize,", text):
        size = text[m.end():text.index(";", m.end())]
        assert not re.search(r"\bsmem\b", size), size
