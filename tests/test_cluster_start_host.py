"""Sources of the kernels that touch another CTA's shared memory: that is allowed once the other CTA is known to run, so a barrier of the whole cluster stands in front
of the first such access."""
import re

import pytest
from test_dependency_wait_host import CSRC, kernels

# functions that form a peer's address or reach its memory, in the files that have them
HELPERS = set()
for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
    text = path.read_text()
    for m in re.finditer(r"__device__ __forceinline__ \w+ (\w+)\(", text):
        body = text[m.end():text.index("\n}", m.end())]
        if "mapa.shared" in body:
            HELPERS.add(m.group(1))
REMOTE = re.compile(r"mapa\.shared|[sl][td]\.shared::cluster|\b(?:%s)\(" % "|".join(sorted(HELPERS)))
SYNC = re.compile(r"barrier\.cluster\.wait|\b\w+_cluster_sync\(\)")
PEERS = [k for k in kernels() if REMOTE.search(k[3])]


def test_the_kernels_are_found():
    assert len(HELPERS) >= 5 and {"few_attn_kernel", "latent_decode_kernel", "linear_sum_kernel"} <= {k[1] for k in PEERS}


@pytest.mark.parametrize("kernel", PEERS, ids=lambda k: f"{k[0]}-{k[1][:40]}")
def test_a_cluster_barrier_stands_in_front(kernel):
    first = SYNC.search(kernel[3])
    assert first is not None and first.start() < REMOTE.search(kernel[3]).start()
