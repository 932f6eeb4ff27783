"""Kernels that overlap their predecessor on the stream, read from the sources: each waits for it, and tensor memory is
taken after that wait and before the successor is let in (a block that holds some while it waits, beside a block of its
predecessor that has yet to take its own, would stop both for good)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "slang_b200", "csrc")


def _kernels():
    """(name, body) of every __global__ function of the sources, comments left out."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            head = text[a:text.index("{", a)]
            name = [n for n in re.findall(r"(\w+)\s*\(", head) if n != "__launch_bounds__"][0]
            depth, i = 0, text.index("{", a)
            for j in range(i, b):
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                if depth == 0:
                    break
            out.append((name, text[i:j + 1]))
    return out


OVERLAPPING = [(n, b) for n, b in _kernels() if "grid_release()" in b or "grid_wait()" in b]


def test_the_overlapping_kernels_are_found():
    names = {n for n, _ in OVERLAPPING}
    assert {"learn_gradient_narrow_kernel", "forward_narrow_kernel", "forward_tc_kernel", "learn_gradient_simt_kernel",
            "adjust_parameters_kernel", "learnGradient", "learnGradient_coopvec", "adjustParameters"} <= names


@pytest.mark.parametrize("name,body", OVERLAPPING, ids=[n for n, _ in OVERLAPPING])
def test_tensor_memory_between_wait_and_release(name, body):
    assert body.count("grid_wait()") == 1
    if "tmem_alloc(" not in body:
        return
    take = body.index("tmem_alloc(")
    assert body.index("grid_wait()") < take
    releases = [m.start() for m in re.finditer(r"grid_release\(\)", body)]
    # (a build without tensor memory may release at once)
    late = [r for r in releases if not body[:r].rstrip().endswith("if constexpr (!kSlots)")]
    assert len(late) == 1 and late[0] > take
    assert "}" not in body[take:late[0]]   # by the warp that took it
