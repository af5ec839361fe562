"""Distributed shared memory may be touched only once every CTA of the cluster has started, which a
cluster barrier guarantees and the time that a kernel's first loads take does not.  Read from the
kernels' source, since a missing barrier is not something to run."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gap_b200", "csrc")
BARRIER = re.compile(r"\bcta\.sync\(\)|this_cluster\(\)\.sync\(\)")


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            if "map_shared_rank" in text[a:b]:
                yield os.path.basename(path), text[a:b]


def test_cluster_barrier_before_the_first_remote_access():
    found = list(_kernels())
    assert len(found) == 2  # k_dense_solve_cl, k_nr_small
    for name, body in found:
        first = BARRIER.search(body)
        assert first and first.start() < body.index("map_shared_rank"), name
