"""Kernels that start before their predecessor has ended: what their sources have to keep to, read from the sources (a kernel that
breaks these rules may hang, so the rules are not tried out on a GPU)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xinfer_b200", "csrc")


def _without_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", " ", text, flags=re.S)


def _block(text, at):
    """The text between the brace that opens at or behind ``at`` and the one that closes it."""
    begin = text.index("{", at)
    depth = 0
    for i in range(begin, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[begin + 1:i]
    raise AssertionError("unbalanced braces")


def kernels_of(path):
    """(name, parameters, body) of every kernel that the file defines."""
    text = _without_comments(open(path).read())
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i - 1], _block(text, i)


FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
ALLOC = re.compile(r"tcgen05\.alloc|\btmem_alloc\s*\(")


def test_the_kernels_are_found():
    found = [name for f in FILES for name, _, _ in kernels_of(f)]
    assert len(found) == sum(len(re.findall(r"__global__\s+void", _without_comments(open(f).read()))) for f in FILES)
    assert sum(bool(ALLOC.search(body)) for f in FILES for _, _, body in kernels_of(f)) >= 6


@pytest.mark.parametrize("path", [f for f in FILES if ALLOC.search(open(f).read())], ids=os.path.basename)
def test_successors_start_only_once_tensor_memory_is_allocated(path):
    # A successor's blocks may allocate tensor memory and hold it until this grid has ended.
    for name, _, body in kernels_of(path):
        alloc = ALLOC.search(body)
        if alloc is None:
            continue
        allocated = body.index("__syncthreads()", alloc.start())
        starts = [m.start() for m in re.finditer(r"pdl_(launch_dependents|overlap_few)\(\)", body)]
        assert starts, name
        for at in starts:
            leaves = re.match(r"pdl_launch_dependents\(\);\s*pdl_wait\(\);\s*return;", body[at:])
            assert at > allocated or leaves, f"{name} lets its successor start before it has allocated tensor memory"
