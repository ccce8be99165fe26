"""Distributed shared memory may be accessed only once the target CTA has started, which a cluster barrier that every
CTA passes at the kernel's start guarantees. Read from the source: each kernel that reaches another CTA's shared memory
passes such a barrier, outside any branch or loop, before its first access."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "modlin-rs_b200", "csrc")
BARRIER = re.compile(r"\b(?:this_cluster\s*\(\s*\)|cl)\s*\.\s*sync\s*\(\s*\)|\bcluster_sync_all\s*\(\s*\)")
REMOTE = re.compile(r"\b(?:map_shared_rank|cluster_addr)\b")


def kernels(name):
    """(kernel name, body without comments) of every __global__ function with a body."""
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"__global__(?:\s+void|\s+__launch_bounds__\s*\([^)]*\))*\s+(\w+)\s*\([^{;]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i - 1]


def first_barrier(body):
    """Where the first unconditional cluster barrier stands, or None."""
    for m in BARRIER.finditer(body):
        if body.count("{", 0, m.start()) == body.count("}", 0, m.start()):
            return m.start()
    return None


@pytest.mark.parametrize("name,kernel", [("rank_batch_team.cu", "rank_team_kernel"),
                                         ("rank_tc.cu", "trailing_tc_pair_kernel")])
def test_barrier_before_the_first_remote_access(name, kernel):
    body = dict(kernels(name))[kernel]
    use = REMOTE.search(body)
    assert use is not None
    barrier = first_barrier(body)
    assert barrier is not None and barrier < use.start()
