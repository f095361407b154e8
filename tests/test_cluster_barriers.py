"""Distributed shared memory by the programming model, read off the kernels' source (a missing barrier shows in no
result: it takes a CTA that starts late, or a warp that lags). A CTA's shared memory may be touched by the others of its
cluster only once it is known to run, which a cluster barrier establishes."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lapstack_b200", "csrc")


def _code(name):
    """A source file without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _body(text, kernel):
    """The text between the braces of a kernel's definition."""
    at = text.index("{", re.search(r"\b%s\(" % kernel, text).end())
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError(kernel)


def _kernels_with_remote_memory():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = _code(name)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^()]*(?:\([^()]*\)[^()]*)*\)\s*)?(\w+)\(", text):
            if "map_shared_rank" in _body(text[m.start():], m.group(1)):
                found.append((name, m.group(1)))
    return found


def test_the_cluster_kernels_are_found():
    assert _kernels_with_remote_memory() == [("lsb_align.cu", "nm_cluster_kernel"), ("lsb_wls.cu", "coarse_h_kernel")]


# where each kernel first touches another CTA's shared memory
FIRST_REMOTE = {"nm_cluster_kernel": r"\*cl\.map_shared_rank\(", "coarse_h_kernel": r"\bput\(0,"}


@pytest.mark.parametrize("kernel", sorted(FIRST_REMOTE))
def test_a_cluster_barrier_comes_before_the_first_remote_access(kernel):
    name = {k: n for n, k in _kernels_with_remote_memory()}[kernel]
    body = _body(_code(name), kernel)
    first = re.search(FIRST_REMOTE[kernel], body).start()
    assert "cl.sync()" in body[:first], "another CTA's shared memory is written before the cluster is known to run"


def _after_level_loop_starts(kernel):
    body = _body(_code("lsb_align.cu"), kernel)
    loop = re.search(r"for \(int L = [^)]*\)", body)
    return body[loop.end():]


@pytest.mark.parametrize("kernel", ["nm_search_kernel", "nm_cluster_kernel"])
def test_a_search_level_begins_behind_a_barrier(kernel):
    """Warp 0 writes `pending` for the next level; every other warp has left the loop before, which reads it, only behind
    a barrier of the CTA."""
    rest = _after_level_loop_starts(kernel)
    assert "while (pending > 0)" in rest
    assert "__syncthreads();" in rest[:rest.index("pending =")], "a warp may still be reading the last level's count"
