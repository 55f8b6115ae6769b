"""Shared memory of another block of a cluster: a kernel may touch it only once every block of
the cluster has started, which a cluster barrier before the first access ensures."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "gain-mpi_gb300", "csrc")


def _body(src, at):
    """The brace-balanced block that opens at or after position `at`."""
    i = src.index("{", at)
    depth = 0
    for k in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        if depth == 0:
            return src[i:k]
    raise AssertionError("unbalanced braces")


def test_a_cluster_barrier_precedes_every_remote_shared_memory_access():
    kernels = 0
    for name in sorted(os.listdir(SRC)):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(SRC, name)).read())
        for m in re.finditer(r"__global__", src):
            body = _body(src, m.end())
            remote = [body.find(w) for w in ("map_shared_rank", "cluster_map(") if w in body]
            if not remote:
                continue
            kernels += 1
            barrier = [body.find(w) for w in ("barrier_wait(", "cluster_sync_all()", ".sync()") if w in body]
            assert barrier and min(barrier) < min(remote), (name, src[m.start():m.start() + 120])
    assert kernels >= 2      # the dot product and the CTA-pair GEMMs
