"""The tcgen05 forward kernels where their work items are at their smallest and most uneven, and at head_dim 64.

A CTA walks over many items, prefetches the next one and stores an item's output behind its back, so the lists here mix
lengths from zero to the whole grid; the calls on fewer SMs give every CTA four of them.  Tolerance against the fp32
oracle: rel-L2 <= 1e-2 in bf16 and 1.3e-3 in fp16 (P is rounded to the input type, 2^-9 and 2^-12 relative, before the
second contraction).  Log-sum-exp of two kernels: 1e-3 absolute; a score is an fp32 sum of up to 128 products of unit
variance, at most 128 * 2^-24 * 128 * 0.09 = 1e-4 off whatever the order, and the sums of the probabilities add less.
"""
import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B
from longcat_video_b200.synthetic import Workload, make_qkv
from oracle import bsa_oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

TC = {128: L.ATTN_TC, 64: L.ATTN_AUTO}  # the head_dim 64 form is only reached by AUTO
TOL = {torch.bfloat16: 1e-2, torch.float16: 1.3e-3}

# name: (batch, heads, head_dim, grid_q, grid_k, block, dtype)
SHAPES = {
    "d64_bf16": (1, 3, 64, (4, 8, 12), (8, 8, 12), (4, 4, 4), torch.bfloat16),          # odd number of query blocks per head
    "d64_fp16_batch2": (2, 2, 64, (8, 8, 8), (8, 8, 8), (4, 4, 4), torch.float16),
    "d64_fp16_ragged": (1, 2, 64, (5, 7, 9), (6, 7, 10), (4, 4, 4), torch.float16),
    "d64_block248": (1, 2, 64, (4, 8, 16), (4, 8, 16), (2, 4, 8), torch.bfloat16),
    "d64_items": (1, 12, 64, (8, 16, 24), (4, 8, 8), (4, 4, 4), torch.bfloat16),        # 288 items: two for most CTAs
    "d128_items": (1, 12, 128, (8, 16, 24), (4, 8, 8), (4, 4, 4), torch.bfloat16),
    "d128_items_ragged": (1, 10, 128, (8, 15, 23), (4, 7, 9), (4, 4, 4), torch.bfloat16),
    "blocks128_items": (1, 14, 128, (8, 16, 24), (4, 8, 16), (4, 4, 8), torch.bfloat16),  # 336 items of one block
    "blocks128_items_fp16": (1, 14, 128, (8, 15, 24), (4, 7, 16), (4, 4, 8), torch.float16),
}


# 336 items (84 CTAs below), key grids of 56 and more blocks (128-token blocks: 36): lists that span several windows of sixteen (128-token blocks: thirty-two) entries, and
# rings of K, V and, on ragged grids, key masks that turn over several times within an item.
LONG = {
    "long_d64_bf16": (1, 14, 64, (8, 16, 24), (8, 16, 28), (4, 4, 4), torch.bfloat16),
    "long_d64_fp16": (2, 7, 64, (8, 16, 24), (8, 16, 32), (4, 4, 4), torch.float16),
    "long_d64_ragged_bf16": (1, 14, 64, (8, 15, 23), (8, 15, 27), (4, 4, 4), torch.bfloat16),
    "long_d64_ragged_fp16": (1, 14, 64, (7, 11, 30), (7, 15, 27), (2, 4, 8), torch.float16),
    "long_d128": (1, 14, 128, (8, 16, 24), (8, 16, 28), (4, 4, 4), torch.bfloat16),
    "long_d128_ragged": (1, 14, 128, (8, 15, 23), (8, 15, 27), (4, 4, 4), torch.float16),
    "long_blocks128": (1, 14, 128, (8, 16, 24), (8, 24, 24), (4, 4, 8), torch.bfloat16),
    "long_blocks128_ragged": (1, 14, 128, (8, 16, 23), (8, 23, 23), (4, 4, 8), torch.float16),
}


@pytest.fixture
def fewer_sms():
    """The persistent kernels leave as many SMs idle as the library allows: 84 CTAs on a B200."""
    old = L.lib().lcbsa_set_attn_sm_reserve(64)
    assert old >= 0
    yield
    assert L.lib().lcbsa_set_attn_sm_reserve(old) == 64


@pytest.mark.parametrize("name", sorted(LONG))
def test_many_items_per_cta_and_long_lists(name, fewer_sms):
    _check_uneven(name, 9300 + sorted(LONG).index(name), LONG[name], "mixed")


@pytest.mark.parametrize("lists", ["short", "mixed"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_uneven_lists(name, lists):
    _check_uneven(name, 9100 + sorted(SHAPES).index(name), SHAPES[name], lists)


def _check_uneven(name, seed, shape, lists):
    b, h, d, gq, gk, chunk, dt = shape
    wl = Workload(name, seed, b, h, d, gq, gk, chunk, 0.5, dt, "normal")
    q, k, v = make_qkv(wl)
    nq, nk = O.num_blocks(gq, chunk), O.num_blocks(gk, chunk)
    gen = torch.Generator().manual_seed(wl.seed)
    cap = nk
    cnt = torch.randint(0, min(3, cap + 1) if lists == "short" else cap + 1, (b, h, nq), generator=gen).to(torch.int32)
    idx = torch.full((b, h, nq, cap), -1, dtype=torch.int32)
    for i, c in enumerate(cnt.flatten().tolist()):
        if c:
            idx.view(-1, cap)[i, :c] = torch.sort(torch.randperm(nk, generator=gen)[:c]).values.to(torch.int32)
    ref, ref_lse = O.attention(q, k, v, gq, gk, chunk, chunk, idx, cnt)
    out, lse = B.attn_fwd_bsa_varlen(q.cuda(), k.cuda(), v.cuda(), 1 / d ** 0.5, idx.cuda(), cnt.cuda(), gq, gk, chunk, chunk,
                                     return_lse=True, impl=TC[d])
    L.check(L.lib().lcbsa_check_device_status())
    assert torch.isfinite(out.float()).all()
    assert rel_l2(out.float().cpu(), ref) <= TOL[dt]
    # the warp-level kernel serves every shape: the same rows are empty, and the same log-sum-exp to fp32 accuracy
    other, other_lse = B.attn_fwd_bsa_varlen(q.cuda(), k.cuda(), v.cuda(), 1 / d ** 0.5, idx.cuda(), cnt.cuda(), gq, gk, chunk, chunk,
                                             return_lse=True, impl=L.ATTN_MMA)
    full = torch.isfinite(other_lse)
    assert torch.equal(full, torch.isfinite(lse))
    assert float((lse - other_lse)[full].abs().max()) <= 1e-3
    assert rel_l2(out.float(), other.float()) <= TOL[dt]


# growth of the scores from one block to the next, as a multiple of what moves the reference between two rounds of a warpgroup
@pytest.mark.parametrize("steep", [1, 4])
@pytest.mark.parametrize("gk", [(4, 16, 16), (4, 15, 15)], ids=["whole", "ragged"])
@pytest.mark.parametrize("d,chunk", [(64, (4, 4, 4)), (128, (4, 4, 4)), (128, (4, 4, 8))], ids=["d64", "d128", "blocks128"])
def test_growing_maximum_rescales(d, chunk, gk, steep):
    """Key blocks whose scores grow by more than 2^8 from one round of a warpgroup to its next: every round moves the reference
    maximum and rescales what has been accumulated.  One coordinate carries the growth (a step per block that bf16 holds
    exactly), the others carry scores of a quarter of the usual spread."""
    gq = (4, 8, 8)
    wl = Workload("grow", 9200 + d, 1, 2, d, gq, gk, chunk, 0.0, torch.bfloat16, "normal")
    q, k, v = make_qkv(wl)
    nq, nk = O.num_blocks(gq, chunk), O.num_blocks(gk, chunk)
    bs = chunk[0] * chunk[1] * chunk[2]
    # a warpgroup takes every second block of 64 tokens, and one of the two halves of every block of 128
    per_round = 2 if bs == 64 else 1
    step = {64: 28.0, 128: 36.0}[d] * (2 // per_round) * steep  # 5.0 and 4.6 (2^...) per block of 64 tokens
    tm = O.token_map(gk, chunk).long()
    order = torch.empty(gk[0] * gk[1] * gk[2])
    order[tm[tm >= 0]] = torch.arange(nk).repeat_interleave(bs)[tm.flatten() >= 0].float()
    q, k = (0.25 * q).to(q.dtype), k.clone()
    q[..., 0] = 1.0
    k[..., 0] = (step * order).to(k.dtype)
    log2_scores = torch.einsum("bhqd,bhkd->bhqk", q.float(), k.float()) * d ** -0.5 * 1.4427
    top = torch.stack([log2_scores[..., order == n].amax(-1) for n in range(nk)], -1)
    assert float((top[..., per_round:] - top[..., :-per_round]).min()) > 8.0
    idx = torch.arange(nk, dtype=torch.int32).expand(1, 2, nq, nk).contiguous()
    cnt = torch.full((1, 2, nq), nk, dtype=torch.int32)
    ref, _ = O.attention(q, k, v, gq, gk, chunk, chunk, idx, cnt)
    out = B.attn_fwd_bsa_varlen(q.cuda(), k.cuda(), v.cuda(), 1 / d ** 0.5, idx.cuda(), cnt.cuda(), gq, gk, chunk, chunk, impl=TC[d])
    L.check(L.lib().lcbsa_check_device_status())
    assert rel_l2(out.float().cpu(), ref) <= TOL[torch.bfloat16]
