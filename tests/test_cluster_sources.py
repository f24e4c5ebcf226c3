"""The kernels' sources: a CTA may touch the shared memory of another CTA of its cluster only once that one is known to run, that is behind a cluster barrier."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vllm_neuron_b200", "csrc")
BARRIER = re.compile(r"\bcluster_wait\(\)|\bcluster_sync_all\(\)")


def _kernels_that_reach_into_peers():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        starts = [m.start() for m in re.finditer(r"\b__global__\b", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            end = text.find("\n}\n", a)
            body = text[a:b if end < 0 else min(end, b)]
            if "mapa_shared(" in body:
                yield pytest.param(body, id=f"{name}:{re.search(r'(\w+_kernel)', body).group(1)}")


@pytest.mark.parametrize("body", list(_kernels_that_reach_into_peers()))
def test_a_cluster_barrier_stands_before_the_first_access_to_a_peer(body):
    barrier = BARRIER.search(body)
    assert barrier, "no cluster barrier"
    assert barrier.start() < body.index("mapa_shared(")
