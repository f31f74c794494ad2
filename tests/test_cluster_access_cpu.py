"""Thread-block clusters: distributed shared memory is accessed only between cluster barriers.

A block of a cluster may be written to or read from by another one only once it has started,
which a launch attribute does not promise and a cluster barrier does, and only until it
leaves.  Every kernel that maps another block's shared memory is read here as text: a barrier
(sync, or the wait of an arrive) stands before its first access and one after its last."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda_3d_gb300", "csrc")
BARRIER = re.compile(r"cluster\.(sync|barrier_wait)\s*\(")
ACCESS = re.compile(r"map_shared_rank\s*\(")


def cluster_kernels():
    """(file, kernel, body) of every kernel that maps another block's shared memory"""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\(", text):
            head = re.compile(r"[{;]").search(text, m.end())
            if not head or head.group() == ";":
                continue  # a declaration
            start = end = head.start()
            depth = 0
            while depth or end == start:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            body = text[start:end]
            if ACCESS.search(body):
                yield name, m.group(1), body


def test_kernels_are_found():
    assert {k for _, k, _ in cluster_kernels()} >= {"k_cluster_sort", "k_icp_finalize"}


@pytest.mark.parametrize("name,kernel,body", list(cluster_kernels()), ids=lambda v: v if len(v) < 40 else "")
def test_remote_accesses_lie_between_barriers(name, kernel, body):
    access = [m.start() for m in ACCESS.finditer(body)]
    barrier = [m.start() for m in BARRIER.finditer(body)]
    assert barrier and barrier[0] < access[0], f"{name}: {kernel} accesses a block that may not have started"
    assert barrier[-1] > access[-1], f"{name}: {kernel} accesses a block that may have left"


def test_every_context_asks_for_the_one_launch_sort_itself():
    """whether the device runs the cluster's kernels is kept in the context, not in the process:
    one context that could not set them up must not decide for those after it"""
    with open(os.path.join(CSRC, "cloud.cu")) as f:
        text = f.read()
    body = text[text.index("int gca3d_create("):text.index("int gca3d_destroy(")]
    assert "grid_cluster_enable() && voxel_cluster_enable()" in body
    assert "call_once" not in text and "static bool ok" not in text
