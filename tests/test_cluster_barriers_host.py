"""Shared memory of another CTA of the cluster exists from the moment that CTA has
started: a kernel that reaches for it (map_shared_rank) has met the cluster's barrier
before, and meets it again before a CTA may leave. Read from the sources, since the
values of a run show neither."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WAIT = re.compile(r"\.(sync|barrier_wait)\(")


def kernels_with_remote_shared_memory():
    for path in sorted(glob.glob(os.path.join(ROOT, "truepix_b200", "csrc", "*.cu*"))):
        text = open(path).read()
        for m in re.finditer(r"\n__global__[^;{]*\{(.*?)\n\}", text, re.S):
            if "map_shared_rank" in m.group(1):
                yield os.path.basename(path), m.group(1)


def test_barrier_on_both_sides_of_a_remote_access():
    found = list(kernels_with_remote_shared_memory())
    assert found
    for name, body in found:
        first, last = body.index("map_shared_rank"), body.rindex("map_shared_rank")
        assert WAIT.search(body[:first]), name
        assert WAIT.search(body[last:]), name
