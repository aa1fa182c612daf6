"""The cdf selector on both sides of every row length at which its sorting network changes, bit for bit against the oracle."""
import pytest
import torch

from longcat_video_b200.block_sparse_attention import bsa_interface as B
from oracle import bsa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nk", [511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049])
def test_row_lengths_around_the_network_widths(nk, dtype):
    g = torch.Generator().manual_seed(nk)
    q = torch.randn(1, 2, 5, 128, generator=g).to(dtype)
    k = (torch.randn(1, 2, nk, 128, generator=g) * 0.7).to(dtype)
    k[:, :, 1::7] = k[:, :, :1]  # equal scores: the order among them is by index
    idx, cnt = B.get_select_indices_from_pooled(q.cuda(), k.cuda(), None, 0.7)
    want_idx, want_cnt = O.cdf_select(O.score(q, k), 0.7, 1 / 128 ** 0.5, 0)
    assert torch.equal(cnt.cpu(), want_cnt) and torch.equal(idx.cpu(), want_idx)
