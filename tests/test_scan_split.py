"""Which requests of a step run a recurrence in chunks: those whose own portion is long, whatever else the step holds."""
from types import SimpleNamespace

import pytest

from railgun_b200 import ops


@pytest.mark.parametrize("lengths,least,want", [
    ([1] * 32, 192, (0, True)), ([191], 192, (0, True)), ([192], 192, (3, False)), ([1, 200, 1, 193], 192, (8, True)),
    ([512, 511], 512, (8, True)), ([513, 2048], 512, (41, False)), ([1] * 32 + [128], 192, (0, True))])
def test_by_each_requests_own_portion(lengths, least, want):
    assert ops.scan_split(SimpleNamespace(max_query_len=max(lengths), layout=(tuple(lengths), 0, ())), least) == want


def test_a_static_batch_of_single_tokens_has_no_layout():
    assert ops.scan_split(SimpleNamespace(max_query_len=1, layout=()), ops.DECAY_CHUNK_MIN_TOKENS) == (0, True)
