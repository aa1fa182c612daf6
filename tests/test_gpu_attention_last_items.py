"""The last items of a CTA, one block long each: the result of the last is staged where the store of the one before is still read.

Every query block lists one key block; the check is against the fp32 oracle, rel-L2 <= 1e-2 (bf16 probabilities).  84 CTAs, two or
three items each, five calls: the order in which stores and merges meet differs from call to call."""
import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B
from longcat_video_b200.synthetic import Workload, make_qkv
from oracle import bsa_oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# (heads, head_dim, grid_q, grid_k, block): 192 and 240 items on 84 CTAs
SHAPES = {"d128": (8, 128, (8, 16, 24), (4, 8, 8), (4, 4, 4)), "d64": (8, 64, (8, 16, 24), (4, 8, 8), (4, 4, 4)),
          "ragged": (8, 128, (8, 15, 23), (4, 7, 9), (4, 4, 4)), "blocks128": (10, 128, (8, 16, 24), (4, 8, 16), (4, 4, 8))}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_items_of_one_block(name):
    h, d, gq, gk, chunk = SHAPES[name]
    wl = Workload(name, 9700 + sorted(SHAPES).index(name), 1, h, d, gq, gk, chunk, 0.5, torch.bfloat16, "normal")
    q, k, v = make_qkv(wl)
    nq, nk = O.num_blocks(gq, chunk), O.num_blocks(gk, chunk)
    gen = torch.Generator().manual_seed(wl.seed)
    idx = torch.randint(0, nk, (1, h, nq, 1), generator=gen).to(torch.int32)
    cnt = torch.ones(1, h, nq, dtype=torch.int32)
    scale = 1 / d ** 0.5
    ref, _ = O.attention(q, k, v, gq, gk, chunk, chunk, idx, cnt)
    old = L.lib().lcbsa_set_attn_sm_reserve(64)
    try:
        assert old >= 0
        args = [t.cuda() for t in (q, k, v)]
        lists = [t.cuda() for t in (idx, cnt)]
        for _ in range(5):
            out = B.attn_fwd_bsa_varlen(*args, scale, *lists, gq, gk, chunk, chunk)
            assert rel_l2(out.float().cpu(), ref) <= 1e-2
    finally:
        L.lib().lcbsa_set_attn_sm_reserve(old)
