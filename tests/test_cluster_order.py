"""Kernels that run in clusters: a block's shared memory is another's to read only once every block of the cluster
has started, which a cluster barrier's completion says, and until none may have left, which the last one's says.
The order stands in the source, where this reads it: no wrong byte need show when it is broken."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "artful_gb300", "csrc")
ARRIVE = re.compile(r"cluster\.sync\(\)|barrier\.cluster\.arrive")
WAIT = re.compile(r"cluster\.sync\(\)|barrier\.cluster\.wait")
REMOTE = re.compile(r"map_shared_rank|\bmapa\b|shared::cluster")


def _cluster_kernels():
    """The name and body of every kernel with cluster dimensions, comments blanked."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = re.sub(r"/\*.*?\*/|//[^\n]*", " ", f.read(), flags=re.S)
        for m in re.finditer(r"__cluster_dims__", text):
            start = text.index("{", m.end())
            depth, at = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
                if depth == 0:
                    break
            yield re.search(r"(\w+)\s*\($", text[:text.index("(const", m.end()) + 1]).group(1), text[start:at]


KERNELS = dict(_cluster_kernels())


def test_the_gas_step_is_a_cluster_kernel():
    assert "gasStep" in KERNELS


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_other_blocks_memory_is_reached_between_cluster_barriers(name):
    body = KERNELS[name]
    reached = [m.start() for m in REMOTE.finditer(body)]
    waits, arrives = [m.start() for m in WAIT.finditer(body)], [m.start() for m in ARRIVE.finditer(body)]
    assert reached and waits and arrives
    assert waits[0] < reached[0], "another block's shared memory is reached before the cluster has started"
    assert arrives[-1] > reached[-1] and waits[-1] > arrives[-1], "a block may leave while its memory is read"
