"""Non-finite inputs: a row with a NaN or an infinite score comes out as NaN, every other row as if nothing had happened.

The reference is a dense softmax in float64 over the keys of a row's list.  rel-L2 of the finite part <= 1e-2 in bf16 and
1.3e-3 in fp16: P is rounded to the input type (2^-9 and 2^-12 relative) before the second contraction.
"""
import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B
from oracle import bsa_oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

TOL = {torch.bfloat16: 1e-2, torch.float16: 1.3e-3}
# head_dim, block, query grid, key grid, dtype: the three tcgen05 forms on whole and on ragged grids
SHAPES = {
    "d64_fp16": (64, (4, 4, 4), (4, 8, 8), (8, 8, 8), torch.float16),
    "d64_ragged": (64, (4, 4, 4), (4, 7, 9), (6, 7, 10), torch.bfloat16),
    "d128": (128, (4, 4, 4), (4, 8, 8), (8, 8, 8), torch.bfloat16),
    "d128_ragged": (128, (4, 4, 4), (4, 7, 9), (6, 7, 10), torch.float16),
    "blocks128": (128, (4, 4, 8), (4, 8, 16), (8, 8, 16), torch.bfloat16),
    "blocks128_ragged": (128, (4, 4, 8), (4, 7, 16), (6, 7, 13), torch.bfloat16),
}


def _case(name):
    d, chunk, gq, gk, dt = SHAPES[name]
    g = torch.Generator().manual_seed(sorted(SHAPES).index(name))
    q, k, v = (torch.randn(1, 2, s[0] * s[1] * s[2], d, generator=g).to(dt) for s in (gq, gk, gk))
    nq, nk = O.num_blocks(gq, chunk), O.num_blocks(gk, chunk)
    idx = torch.arange(nk, dtype=torch.int32).expand(1, 2, nq, nk).contiguous()
    cnt = torch.full((1, 2, nq), nk, dtype=torch.int32)
    cnt[0, 1, :3] = torch.tensor([0, 1, 2])  # an empty list, and lists that only one warpgroup or each of them sees once
    return d, chunk, gq, gk, dt, q, k, v, idx, cnt


def _tokens(grid, chunk, block):
    t = O.token_map(grid, chunk)[block].long()
    return t[t >= 0]


def _dense(q, k, v, gq, gk, chunk, idx, cnt):
    out = torch.zeros(q.shape, dtype=torch.float64)
    for h in range(q.shape[1]):
        for b in range(idx.shape[2]):
            rows = _tokens(gq, chunk, b)
            n = int(cnt[0, h, b])
            if n == 0:
                continue
            keys = torch.cat([_tokens(gk, chunk, int(j)) for j in idx[0, h, b, :n]])
            s = (q[0, h, rows].double() @ k[0, h, keys].double().T) * q.shape[-1] ** -0.5
            p = torch.softmax(s, -1)
            p[s.amax(-1) == float("-inf")] = 0.0  # no key at all: a row of zeros
            out[0, h, rows] = p @ v[0, h, keys].double()
    return out


def _compare(q, k, v, gq, gk, chunk, idx, cnt, dt):
    want = _dense(q, k, v, gq, gk, chunk, idx, cnt)
    lse = {}
    for impl in (L.ATTN_AUTO, L.ATTN_MMA):
        got, lse[impl] = B.attn_fwd_bsa_varlen(q.cuda(), k.cuda(), v.cuda(), q.shape[-1] ** -0.5, idx.cuda(), cnt.cuda(), gq, gk, chunk,
                                               chunk, return_lse=True, impl=impl)
        L.check(L.lib().lcbsa_check_device_status())
        got = got.double().cpu()
        assert torch.equal(torch.isnan(got), torch.isnan(want)), impl
        assert torch.equal(torch.isinf(got), torch.isinf(want)), impl
        fin = torch.isfinite(want)
        assert rel_l2(got[fin], want[fin]) <= TOL[dt], impl
    assert torch.equal(torch.isfinite(lse[L.ATTN_AUTO]), torch.isfinite(lse[L.ATTN_MMA]))
    return want


@pytest.mark.parametrize("where", ["nan_key", "nan_query", "inf_key", "minus_inf_query", "nan_value", "inf_value"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_nan_and_inf_reach_the_rows_they_belong_to(name, where):
    d, chunk, gq, gk, dt, q, k, v, idx, cnt = _case(name)
    val = float("nan") if where.startswith("nan") else float("-inf") if where.startswith("minus") else float("inf")
    # one token of a whole block and one of the last (possibly partial) block
    if where.endswith("query"):
        q[0, 0, 5, 3] = q[0, 1, -1, 4] = val
    elif where.endswith("key"):
        k[0, 0, 5, 3] = k[0, 1, -1, 4] = val
    else:
        v[0, 0, 5, 3] = v[0, 1, -1, 4] = val
    want = _compare(q, k, v, gq, gk, chunk, idx, cnt, dt)
    assert not torch.isfinite(want).all() and torch.isfinite(want).any()


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_blocks_of_minus_inf_scores_leave_no_reference(name):
    """The first two blocks of every list score -inf throughout, the others far below zero: whatever stands in for the
    missing maximum of the first two must not be taken for a score (the rest would underflow against it)."""
    d, chunk, gq, gk, dt, q, k, v, idx, cnt = _case(name)
    q[..., 0] = 1.0
    k[..., 0] = -3000.0
    for block in (0, 1):
        k[:, :, _tokens(gk, chunk, block), 0] = float("-inf")
    want = _compare(q, k, v, gq, gk, chunk, idx, cnt, dt)
    assert torch.isfinite(want).all() and (want[0, 0] != 0).all()
