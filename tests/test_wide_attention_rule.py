"""Which portions of prompts take the tcgen05 attention at head size 128: by their own contexts and by how many blocks there are."""
import pytest

from railgun_b200.parts.attention import wide_attention_pays


@pytest.mark.parametrize("context,tiles,tiles128,nh,nkv,pays", [
    (100, 2, 1, 32, 8, False), (128, 8, 4, 32, 8, False), (256, 4, 2, 32, 8, False), (257, 5, 3, 32, 8, True),
    (129, 5, 3, 32, 8, True), (129, 3, 2, 32, 8, False),                     # 160 blocks of the other kernel are more than 148 SMs
    (128, 2, 1, 32, 32, False), (129, 3, 2, 32, 32, True), (129, 24, 16, 32, 32, False), (256, 8, 5, 32, 32, False),
    (257, 9, 5, 32, 32, True), (2048, 32, 16, 1, 1, True)])
def test_the_rules_edges(context, tiles, tiles128, nh, nkv, pays):
    assert wide_attention_pays(context, tiles, tiles128, nh, nkv, 148) == pays
