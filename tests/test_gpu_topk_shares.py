"""Top-k with few, half, most and all of the keys selected, over scores of either sign: where the search for the threshold starts
depends on the share, the lists do not (exact against the oracle)."""
import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B
from oracle import bsa_oracle as O

pytestmark = pytest.mark.gpu

SPARSITIES = (0.0, 0.01, 0.25, 0.49, 0.5, 0.51, 0.6, 0.9)


def _pooled(kind, dtype, nq, nk, seed):
    """One component that decides the score: its sign and spread per kind."""
    g = torch.Generator().manual_seed(seed)
    qc = torch.zeros(1, 2, nq, 64, dtype=dtype)
    qc[..., 0] = (1.0 + torch.rand(1, 2, nq, generator=g)).to(dtype)
    x = {"both": torch.randn(1, 2, nk, generator=g), "positive": 20.0 + torch.randn(1, 2, nk, generator=g),
         "negative": -20.0 - torch.randn(1, 2, nk, generator=g), "ties": torch.randint(-2, 3, (1, 2, nk), generator=g).float(),
         "equal": torch.full((1, 2, nk), -3.0), "wide": torch.randn(1, 2, nk, generator=g) * 10.0 ** torch.randint(-4, 4, (1, 2, nk), generator=g)}[kind]
    kc = torch.zeros(1, 2, nk, 64, dtype=dtype)
    kc[..., 0] = x.to(dtype)
    return qc, kc


@pytest.mark.parametrize("kind", ["both", "positive", "negative", "ties", "equal", "wide"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nk", [2, 24, 129, 640])
def test_topk_shares(kind, dtype, nk):
    qc, kc = _pooled(kind, dtype, 9, nk, nk)
    for sparsity in SPARSITIES:
        nsel = O.num_selected(sparsity, nk)
        ref, _, _ = O.topk(O.score(qc, kc), nsel)
        idx, cnt = B.get_select_indices_from_pooled(qc.cuda(), kc.cuda(), sparsity)
        assert int(cnt.min()) == int(cnt.max()) == nsel
        assert torch.equal(idx.cpu()[..., :nsel], ref[..., :nsel]), sparsity


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sparsity", SPARSITIES)
def test_topk_shares_of_a_first_part(dtype, sparsity):
    """Rows of the first part select among its keys alone, the others among all."""
    hw, period, split = 6, 5, 2
    n = hw * period
    qc, kc = _pooled("both", dtype, n, n, 5)
    idx, cnt = B.get_select_indices_from_pooled_split(qc.cuda(), kc.cuda(), sparsity, hw, period, split, hw, period, split)
    idx, cnt, first = idx.cpu(), cnt.cpu(), hw * split
    for rows, keys in ((slice(0, first), first), (slice(first, n), n)):
        nsel = O.num_selected(sparsity, keys)
        ref, _, _ = O.topk(O.score(qc[:, :, rows].contiguous(), kc[:, :, :keys].contiguous()), nsel)
        assert int(cnt[:, :, rows].min()) == int(cnt[:, :, rows].max()) == nsel
        assert torch.equal(idx[:, :, rows, :nsel], ref[..., :nsel])


def test_the_share_does_not_decide_the_time():
    """Scores of both signs: three quarters of the keys take no longer than the few that the model selects, but for their longer
    lists (about a tenth); with a search that walks down from the largest key they took a fifth longer."""
    g = torch.Generator().manual_seed(1)
    q, k = (torch.randn(1, 32, 624, 64, generator=g).to(torch.float16).cuda() for _ in range(2))

    def shortest(sparsity):
        best = float("inf")
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(300000)  # the launches of the call are queued behind it
            a.record()
            for _ in range(4):
                B.get_select_indices_from_pooled(q, k, sparsity)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    few, many = shortest(0.9375), shortest(0.25)
    L.check(L.lib().lcbsa_check_device_status())
    print(f"624 of 32 heads: 0.9375 {few * 250:.1f} us, 0.25 {many * 250:.1f} us")
    assert many <= 1.16 * few
