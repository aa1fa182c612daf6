"""Tile sizes of the score kernel: lists equal to the oracle's on both sides of each line of its rule, with partial tiles.

The rule counts tiles over the whole call: up to 296 of 32 scores, then up to 444 of 64, else 128.  Lists are exact."""
import pytest
import torch

from longcat_video_b200.block_sparse_attention import bsa_interface as B
from oracle import bsa_oracle as O

pytestmark = pytest.mark.gpu

# (heads, query blocks, key blocks, head_dim): what is launched
SHAPES = {
    "32_smallest": (1, 1, 1, 128),           # two tiles of 32 (the row of keys is padded to 64)
    "32_partial": (3, 33, 65, 64),           # 3 x 2 x 4 = 24
    "32_last": (4, 270, 250, 128),           # 9 x 8 x 4 = 288
    "64_first": (5, 257, 250, 64),           # 9 x 8 x 5 = 360 of 32; 5 x 4 x 5 = 100 of 64
    "64_last": (4, 641, 630, 128),           # 11 x 10 x 4 = 440 of 64
    "128_first": (5, 577, 570, 128),         # 10 x 9 x 5 = 450 of 64; partial tiles of 128 both ways
}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_lists_on_both_sides_of_the_tile_rule(name, dtype):
    h, nq, nk, d = SHAPES[name]
    g = torch.Generator().manual_seed(9800 + sorted(SHAPES).index(name))
    q, k = (torch.randn(1, h, n, d, generator=g).to(dtype) for n in (nq, nk))
    idx, cnt = B.get_select_indices_from_pooled(q.cuda(), k.cuda(), 0.75)
    nsel = O.num_selected(0.75, nk)
    want, want_cnt, _ = O.topk(O.score(q, k), nsel)
    assert torch.equal(cnt.cpu(), want_cnt)
    assert torch.equal(idx.cpu()[..., :nsel], want[..., :nsel])
