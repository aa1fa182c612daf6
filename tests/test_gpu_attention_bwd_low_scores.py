"""Backward on key grids with partial blocks when every score of a row lies far below zero.  A key slot outside the grid has the
score 0, so 2^(0 - lse * log2 e) overflows there from lse = -88 down; its contribution to dQ has to stay zero."""
import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B
from oracle import bsa_backward as OB
from oracle import bsa_oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid_q, grid_k, chunk_q, chunk_k", [
    ((5, 7, 9), (6, 7, 10), (4, 4, 4), (4, 4, 4)),
    ((8, 8, 16), (5, 6, 13), (4, 4, 8), (4, 4, 4)),   # own blocks of 128 query tokens, partial key blocks
    ((5, 7, 9), (4, 8, 8), (4, 4, 4), (4, 4, 4)),     # partial query blocks alone
])
@pytest.mark.parametrize("level", [3.0, 10.0])
def test_gradients_with_all_scores_far_below_zero(monkeypatch, grid_q, grid_k, chunk_q, chunk_k, level):
    """q and k have a common part of opposite sign: scaled scores around -11.3 level^2, that is -102 and -1130."""
    heads, D = 2, 128
    gen = torch.Generator().manual_seed(int(level))
    sq, sk = (g[0] * g[1] * g[2] for g in (grid_q, grid_k))
    q = (0.3 * torch.randn(1, heads, sq, D, generator=gen) + level).to(torch.bfloat16)
    k = (0.3 * torch.randn(1, heads, sk, D, generator=gen) - level).to(torch.bfloat16)
    v, do = (torch.randn(1, heads, s, D, generator=gen).to(torch.bfloat16) for s in (sk, sq))
    idx, cnt, _, _ = O.block_select(q, k, grid_q, grid_k, 0.4, chunk_q, chunk_k)
    qd, kd, vd, dod, idxd, cntd = (t.cuda() for t in (q, k, v, do, idx, cnt))
    o, lse = B.attn_fwd_bsa_varlen(qd, kd, vd, D ** -0.5, idxd, cntd, grid_q, grid_k, chunk_q, chunk_k, return_lse=True)
    assert float(lse.max()) < -88.8
    args = (dod, qd, kd, vd, o, lse, D ** -0.5, idxd, cntd, grid_q, grid_k, chunk_q, chunk_k)
    got = B.attn_bwd_bsa_varlen(*args)
    monkeypatch.setenv("LCBSA_BWD_IMPL", "mma")
    want = B.attn_bwd_bsa_varlen(*args)
    torch.cuda.synchronize()
    L.check(L.lib().lcbsa_check_device_status())
    _, *ref = OB.attention_backward(q, k, v, do, idx, cnt, grid_q, grid_k, chunk_q, chunk_k)
    for name, g, w, r in zip(("dq", "dk", "dv"), got, want, ref):
        assert torch.isfinite(g).all(), name
        # The warp-level kernels mask such keys; both round P, dS and the results at the same places.  The bound is one unit in
        # the last place of bf16, for sums of fp32 products in another order.
        assert float((g.double() - w.double()).norm() / w.double().norm()) <= 2.0 ** -8, name
        # dQ = sum dS_j K_j with sum dS_j = 0: the common part of K cancels, the rounding of dS times that part does not, so dQ is
        # held by the comparison above alone
        assert name == "dq" or rel_l2(g.float().cpu(), r) <= 1e-2, name
