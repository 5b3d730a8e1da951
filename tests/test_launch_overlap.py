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


# Pointers that may be declared __restrict__ in a kernel that waits for its predecessor: weights and what the host sent before the
# step, which no kernel writes; and plain outputs, whose values come from loads behind the wait.
SENT = set("""rows w b b_alpha b_w b_b w_r correction req_of_token table ids positions q_start slots start_pos block_table norm_w inv_freq
              cq_w sink blocks work bw gain wl wr bias bz bx coef taps dt_bias A_log Dv bi bf q_w k_w dense_weight""".split())
OUTPUTS = set("out y o act prep scores alpha div q_out k_cache v_cache cq choice weight gate prodA endB start cache prev_state".split())


@pytest.mark.parametrize("path", [f for f in FILES if re.search(r"pdl_(wait|overlap_few)\(\)", open(f).read())], ids=os.path.basename)
def test_what_a_predecessor_writes_is_not_promised_to_stay(path):
    # A pointer to const with __restrict__ says that its data does not change while the kernel runs, and one that is read and
    # written that nobody else does: their loads may then be moved in front of the wait.
    for name, params, body in kernels_of(path):
        if not re.search(r"pdl_(wait|overlap_few)\(\)", body):
            continue
        for p in params.split(","):
            if "__restrict__" not in p:
                continue
            word = re.findall(r"\w+", p)[-1]
            if "const" in p.split("*")[0].split():
                ok = word in SENT or (name, word) == ("dyt_kernel", "alpha")
            else:
                ok = word in OUTPUTS
            assert ok, f"{name}: {' '.join(p.split())}"
