"""A CTA's shared memory may be reached from the other CTAs of its cluster only once it is known to have started: in every kernel of a
cluster a barrier of all its CTAs comes before the first store, arrival or copy that reaches another one.  Read from the sources: a run
that meets the fault would be one on memory that is not there yet."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dnet_b200" / "csrc"
REMOTE = re.compile(r"\b(dsmem_st|mbar_arrive_cluster|tma_load_2d_pair|tc_commit_pair|tc_mma_pair)\s*\(")


def kernels():
    """(file, name, body) of every __global__ function that reaches into its cluster"""
    out = []
    for path in sorted(CSRC.glob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            at = text.index("{", m.end())
            depth, end = 0, at
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            body = text[at:end]
            if REMOTE.search(body):
                out.append(pytest.param(body, id=f"{path.name}:{m.group(1)}"))
    return out


@pytest.mark.parametrize("body", kernels())
def test_a_cluster_has_started_before_anything_reaches_into_it(body):
    barrier = body.find("cluster_sync()")
    assert 0 <= barrier < REMOTE.search(body).start()


def test_the_kernels_of_clusters_are_found():
    assert {p.id.split(":")[1] for p in kernels()} >= {"k_gemm_tc", "k_attn_prefill_tc", "k_attn_prefill_q"}
