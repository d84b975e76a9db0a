"""Kernels that write into a peer CTA's shared memory first wait until every CTA
of the cluster has started (cluster.cuh); read from the sources, since a missing
wait shows nothing until a CTA is late."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "warp_sph_gpt_gb300" / "csrc"


def _kernel_body(file, name):
    text = re.sub(r"//[^\n]*", "", (CSRC / file).read_text())
    head = re.search(rf"__global__[^;{{]*?\b{name}\s*\([^{{;]*\)\s*{{", text, flags=re.S)
    assert head, f"{name} is not in {file}"
    depth, at = 1, head.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
    return text[head.end():at]


@pytest.mark.parametrize("file,name", [("coupling.cu", "k_interaction_dem"), ("mpnn.cu", "k_loss")])
def test_peers_have_started_before_their_shared_memory_is_written(file, name):
    body = _kernel_body(file, name)
    first = body.index("map_shared_rank")
    assert 0 <= body.find("cluster_started()") < body.find("cluster_wait_started()") < first
    last = max(m.start() for m in re.finditer("map_shared_rank", body))
    assert re.search(r"\.sync\(\)", body[last:])  # and the sums have landed before they are read
