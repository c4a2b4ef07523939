"""Order of remote shared-memory accesses in the kernels that run on clusters of thread blocks, read from the source: a block may touch
another one's shared memory only once it is known that the other has started, and not after it may have left.  So on the way through
each kernel a wait on the cluster's barrier stands in front of the first remote access and behind the last one."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aeon_b200", "csrc")
FUNCTION = re.compile(r"(__device__|__global__)[^;{}]*?\b(\w+)\s*\([^;{}]*\)\s*\{")
EVENT = re.compile(r"\bcluster\s*\.\s*(?P<wait>sync|barrier_wait)\s*\(|(?P<remote>\bmap_shared_rank)\b|\b(?P<call>\w+)\s*(?:<[^<>;(){}]*>)?\s*\(")


def functions(text):
    """Bodies of the device functions and kernels of a source, by name, and the names of the kernels."""
    text = re.sub(r"//[^\n]*|__(launch_bounds|cluster_dims)__\([^()]*\)", "", text)
    bodies, kernels = {}, []
    for m in FUNCTION.finditer(text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        bodies[m.group(2)] = bodies.get(m.group(2), "") + text[m.end():i]
        if m.group(1) == "__global__":
            kernels.append(m.group(2))
    return bodies, kernels


def events(name, bodies, within=()):
    """Waits ("W") and remote accesses ("R") in source order, calls followed."""
    out = []
    for m in EVENT.finditer(bodies[name]):
        if m.group("wait"):
            out.append("W")
        elif m.group("remote"):
            out.append("R")
        elif m.group("call") in bodies and m.group("call") not in within + (name,):
            out += events(m.group("call"), bodies, within + (name,))
    return out


def cluster_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        bodies, kernels = functions(open(path).read())
        for k in kernels:
            if "R" in events(k, bodies):
                yield pytest.param(bodies, k, id=k)


def test_the_kernels_on_clusters_are_found():
    assert {p.id for p in cluster_kernels()} == {"aug_pack_kernel", "jpeg_entropy_spread_kernel", "jpeg_restart_index_kernel"}


@pytest.mark.parametrize("bodies, kernel", list(cluster_kernels()))
def test_remote_accesses_lie_between_waits(bodies, kernel):
    order = "".join(events(kernel, bodies))
    assert order.startswith("W"), "%s touches another block's memory before it waits for the cluster: %s" % (kernel, order)
    assert order.endswith("W"), "%s may touch the memory of a block that has left: %s" % (kernel, order)
