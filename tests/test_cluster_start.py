"""A CTA of a cluster may reach into another's shared memory only once that
one is known to have started, that is after a cluster barrier. In the source
of every kernel that does, a cluster barrier comes before the first such
access (kernels are straight-line up to there)."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "amigo_b200", "csrc")
REMOTE = re.compile(r"\b(at_rank|row_ptr|push_part|map_shared_rank|member_column)\b")
BARRIER = re.compile(r"\bcl\.sync\(\)|\bcsync<\w+>\(cl\)")


def _kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__", text):
            head = text[m.end():text.index("{", m.end())]
            kernel = re.search(r"(\w+)\s*\(\s*(?:DevPlan|DevState|int|const)", head)
            depth, i = 0, text.index("{", m.end())
            start = i
            while True:
                depth += (text[i] == "{") - (text[i] == "}")
                i += 1
                if depth == 0:
                    break
            body = text[start:i]
            if REMOTE.search(body) and "this_cluster" in body:
                yield pytest.param(body, id=kernel.group(1) if kernel else name)


KERNELS = list(_kernels())


def test_the_cluster_kernels_are_found():
    assert {k.id for k in KERNELS} >= {"cluster_front_kernel", "big_chain_panel_kernel",
                                       "big_panel_kernel", "forward_big_kernel",
                                       "backward_big_kernel"}


@pytest.mark.parametrize("body", KERNELS)
def test_barrier_before_the_first_remote_access(body):
    barrier = BARRIER.search(body)
    assert barrier and barrier.start() < REMOTE.search(body).start()
