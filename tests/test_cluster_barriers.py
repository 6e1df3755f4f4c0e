"""Kernels of a thread-block cluster, read as source: the shared memory of
another CTA exists from the moment that CTA has started until it leaves, and
only a cluster barrier says so.  So every such kernel has one before it names
another CTA's shared memory and one as its last statement, both outside any
branch or loop."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opticrcwafdtd_b200", "csrc")


def _strip(src):
    src = re.sub(r"/\*.*?\*/", " ", src, flags=re.S)
    return re.sub(r"//[^\n]*", "", src)


def _kernels(src):
    """(name, body) of each __global__ function of a comment-free source."""
    for m in re.finditer(r"__global__\s+void\b", src):
        o = m.end()
        lb = re.match(r"\s*__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", src[o:])
        o += lb.end() if lb else 0
        name = re.match(r"\s*(\w+)", src[o:]).group(1)
        b = src.index("{", o)
        depth, e = 0, b
        while True:
            depth += {"{": 1, "}": -1}.get(src[e], 0)
            e += 1
            if depth == 0:
                break
        yield name, src[b + 1:e - 1]


def _cluster_kernels():
    out = []
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        for name, body in _kernels(_strip(open(f).read())):
            if "this_cluster" in body:
                out.append((name, body))
    return out


KERNELS = _cluster_kernels()


def test_the_cluster_kernels_are_found():
    assert {n for n, _ in KERNELS} >= {"k_fdfd_factor", "k_fdfd_sweep", "k_fdfd_red"}


@pytest.mark.parametrize("name,body", KERNELS, ids=[n for n, _ in KERNELS])
def test_barrier_before_the_first_and_after_the_last_remote_access(name, body):
    remote = body.index("map_shared_rank")
    depth = 0
    barriers = []   # unconditional cluster barriers: at the body's own level
    for q, c in enumerate(body):
        depth += {"{": 1, "}": -1}.get(c, 0)
        if depth == 0 and body.startswith("cl.sync();", q):
            # a statement of its own, not the body of a condition without braces
            assert body[:q].rstrip()[-1] in ";}", name
            barriers.append(q)
    assert barriers and barriers[0] < remote, f"{name} names another CTA's shared memory before a cluster barrier"
    assert body.rstrip().endswith("cl.sync();"), f"{name} may leave while another CTA still writes to it"
    assert not re.search(r"\breturn\s*;", body[:remote]), name
