"""Blocks of a cluster reach into each other's shared memory only once all of them are known to run."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "railgun_b200" / "csrc" / "kernels"
REACHES = re.compile(r"map_shared_rank\(|mapa_shared\(")
MEETS = re.compile(r"\.sync\(\);|barrier\.cluster\.wait|cluster_sync_all\(\);")


def bodies(text):
    """The kernels of a source file: name and body."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\((?:[^(){}]|\([^()]*\))*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


@pytest.mark.parametrize("path", sorted(KERNELS.glob("*.cu*")), ids=lambda p: p.name)
def test_a_cluster_meets_before_its_blocks_reach_into_each_other(path):
    for name, body in bodies(path.read_text()):
        reach = REACHES.search(body)
        if reach:
            assert MEETS.search(body[:reach.start()]), f"{name}: another block's shared memory before the cluster has met"


def test_the_kernels_that_reach_into_each_other_are_found():
    found = {name for p in KERNELS.glob("*.cu*") for name, body in bodies(p.read_text()) if REACHES.search(body)}
    assert {"argmax_cluster_kernel", "skinny_gemm_kernel", "tc_stream_kernel", "tc_grouped_kernel"} <= found, found
