"""Distributed shared memory is touched only after a cluster-wide barrier: a block may reach another
block's shared memory once that block is known to run, which a barrier of the cluster before the
first access establishes. Read from the sources, as a kernel without it may well work by luck."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "galaxy_formation_gb300", "csrc")


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^;{]*\)\s*{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            if "map_shared_rank" in text[m.end():end]:
                yield pytest.param(text[m.end():end], id=m.group(1))


KERNELS = list(_kernels())


def test_every_cluster_kernel_is_looked_at():
    assert {p.id for p in KERNELS} >= {"k_scan_cluster", "k_small_sort", "k_direct"}


@pytest.mark.parametrize("body", KERNELS)
def test_a_barrier_comes_before_the_first_remote_access(body):
    before = body[:body.index("map_shared_rank")]
    assert re.search(r"cluster\.(sync|barrier_wait)\(", before)
    # a block also stays until its shared memory is no longer reached: no early return before that
    assert not re.search(r"\breturn\b", before)
