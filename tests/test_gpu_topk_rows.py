"""Top-k over rows of every length at which the kernel's register rows change, against the oracle (exact)."""
import pytest
import torch

from longcat_video_b200.block_sparse_attention import bsa_interface as B
from oracle import bsa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk", [1, 63, 64, 65, 255] + [n + i for n in range(128, 1537, 128) for i in (0, 1)])
@pytest.mark.parametrize("distinct", [3, 4000])
def test_topk_row_lengths(nk, distinct):
    """Both sides of every row length at which the top-k kernel changes, with rows full of ties and rows with few."""
    g = torch.Generator().manual_seed(nk)
    nq, d = 9, 64
    qc = torch.zeros(1, 2, nq, d, dtype=torch.bfloat16)
    qc[..., 0] = torch.randint(1, 5, (1, 2, nq), generator=g).to(torch.bfloat16)
    kc = torch.zeros(1, 2, nk, d, dtype=torch.bfloat16)
    kc[..., 0] = (torch.randint(0, distinct, (1, 2, nk), generator=g) - distinct // 2).to(torch.bfloat16)
    for sparsity in (0.0, 0.5, 0.9, 0.99):
        nsel = O.num_selected(sparsity, nk)
        ref_idx, _, _ = O.topk(O.score(qc, kc), nsel)
        idx, cnt = B.get_select_indices_from_pooled(qc.cuda(), kc.cuda(), sparsity)
        assert int(cnt.min()) == int(cnt.max()) == nsel
        assert torch.equal(idx.cpu()[..., :nsel], ref_idx[..., :nsel])
