"""Which kernel takes short portions of prompts, as far as that is decided on the host, and the tiles that go with it."""
import pytest
import torch

from rustinfer_b200.parts import attention_variants as V


@pytest.mark.parametrize("tiles,kv_heads,group,hd,tokens,keys,sooner", [
    (1, 16, 1, 128, 2, 2, False), (16, 16, 1, 128, 2, 2, True), (16, 16, 1, 128, 2, 1002, False), (64, 16, 1, 128, 2, 1002, False),
    (24, 16, 1, 64, 2, 2, True), (16, 4, 8, 64, 8, 1008, False), (16, 2, 4, 128, 16, 80, False), (24, 16, 2, 64, 2, 202, True),
])
def test_many_portions_over_few_keys(tiles, kv_heads, group, hd, tokens, keys, sooner):
    assert V.rows_are_sooner(tiles, kv_heads, group, hd, tokens, keys, True, 148) == sooner


@pytest.mark.gpu
def test_tiles_follow_the_kernel():
    from rustinfer_b200.parts.base import BuildContext
    attend = V.PlainAttend(BuildContext(torch.device("cuda:0"), torch.bfloat16, 64, 16, max_batch_seqs=4), 8, 2, 64, 64)
    rows = attend._tiles.key
    attend.take_exact(torch.zeros(8, 100, device="cuda:0"))
    assert attend.exact and attend._tiles.key != rows
    attend.take_exact(torch.zeros(8, 5000, device="cuda:0"))          # more distances than the tcgen05 kernel has room for
    assert not attend.exact and attend._tiles.key == rows
