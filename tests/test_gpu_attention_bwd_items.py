"""The backward's persistent passes with many items per CTA: lists of very different lengths, empty ones among them (at the start,
in runs, at the end), against the warp-level passes, which the oracle cases hold (tests/test_gpu_attention_bwd.py)."""
import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B
from tests.helpers import grids_of_capture

pytestmark = pytest.mark.gpu


def _lists(gen, heads, nq, nk, cap, empty):
    """Random ascending lists of 0 .. cap entries over all but the last third of the key blocks, those in ``empty`` without any."""
    cnt = torch.randint(0, cap + 1, (1, heads, nq), generator=gen, dtype=torch.int32)
    cnt[:, :, empty] = 0
    order = torch.rand(1, heads, nq, nk, generator=gen)
    order[..., nk - nk // 3:] = 2.0
    idx = order.argsort(-1)[..., :cap]
    keep = torch.arange(cap).view(1, 1, 1, cap) < cnt[..., None]
    idx = torch.where(keep, idx, nk).sort(-1).values
    return torch.where(idx < nk, idx, -1).to(torch.int32).contiguous(), cnt


@pytest.mark.parametrize("grid, block, dtype, cap, bits", [
    ((8, 32, 36), (4, 4, 4), torch.bfloat16, 40, True),    # 432 items of 64 tokens in each pass
    ((8, 32, 36), (4, 4, 4), torch.float16, 1, True),      # lists of one entry or none
    ((7, 31, 34), (4, 4, 4), torch.bfloat16, 7, True),     # partial edge blocks
    ((8, 32, 48), (4, 4, 8), torch.bfloat16, 9, False),    # 288 items of 128 tokens
    ((8, 32, 48), (4, 4, 8), torch.float16, 1, False),
    ((4, 4, 8), (4, 4, 4), torch.bfloat16, 2, True),       # fewer items than SMs
])
def test_many_items_per_cta(monkeypatch, grid, block, dtype, cap, bits):
    heads, D = 3, 128
    gen = torch.Generator().manual_seed(cap + grid[0])
    S = grid[0] * grid[1] * grid[2]
    n = L.grid_plan(grid, block)[1]
    q, k, v, do = (torch.randn(1, heads, S, D, generator=gen).to(dtype).cuda() for _ in range(4))
    empty = sorted({0, n - 1, *range(n // 3, n // 3 + n // 4)}) if n > 8 else []
    idx, cnt = (t.cuda() for t in _lists(gen, heads, n, n, cap, empty))
    o, lse = B.attn_fwd_bsa_varlen(q, k, v, D ** -0.5, idx, cnt, grid, grid, block, block, return_lse=True)
    args = (do, q, k, v, o, lse, D ** -0.5, idx, cnt, grid, grid, block, block)
    got = B.attn_bwd_bsa_varlen(*args)
    again = B.attn_bwd_bsa_varlen(*args)
    monkeypatch.setenv("LCBSA_BWD_IMPL", "mma")
    want = B.attn_bwd_bsa_varlen(*args)
    torch.cuda.synchronize()
    L.check(L.lib().lcbsa_check_device_status())
    for g, a, w in zip(got, again, want):
        assert torch.equal(g, a)
        if bits:
            assert torch.equal(g, w)
        else:  # fp32 sums in another order, rounded to the dtype: one unit in the last place here and there
            err = (g.double() - w.double()).norm() / w.double().norm()
            assert float(err) <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)


@pytest.mark.parametrize("block", [(4, 4, 4), (4, 4, 8)])
def test_reserved_sms_stay_free(block):
    """Each pass launches one CTA per SM less the reserve, and gives the same bits with another number of CTAs."""
    grid, heads, D = (8, 32, 48), 3, 128
    gen = torch.Generator().manual_seed(3)
    S = grid[0] * grid[1] * grid[2]
    n = L.grid_plan(grid, block)[1]
    q, k, v, do = (torch.randn(1, heads, S, D, generator=gen).to(torch.bfloat16).cuda() for _ in range(4))
    idx, cnt = (t.cuda() for t in _lists(gen, heads, n, n, 5, [0, n - 1]))
    o, lse = B.attn_fwd_bsa_varlen(q, k, v, D ** -0.5, idx, cnt, grid, grid, block, block, return_lse=True)
    args = (do, q, k, v, o, lse, D ** -0.5, idx, cnt, grid, grid, block, block)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert heads * n >= sms
    want = B.attn_bwd_bsa_varlen(*args)
    for reserve in (2, 64):
        old = L.lib().lcbsa_set_attn_sm_reserve(reserve)
        try:
            assert old >= 0
            got = B.attn_bwd_bsa_varlen(*args)
            passes = [ctas for name, ctas in grids_of_capture(lambda: B.attn_bwd_bsa_varlen(*args)) if "bwd_tc_kernel" in name]
        finally:
            L.lib().lcbsa_set_attn_sm_reserve(old)
        torch.cuda.synchronize()
        L.check(L.lib().lcbsa_check_device_status())
        assert passes == [sms - reserve] * 2
        for g, w in zip(got, want):
            assert torch.equal(g, w)
