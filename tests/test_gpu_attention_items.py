"""The tcgen05 forward kernels where their work items are at their smallest and most uneven, and at head_dim 64.

A CTA walks over many items, prefetches the next one and stores an item's output behind its back, so the lists here mix
lengths from zero to the whole grid and there are several items per CTA.  Tolerance against the fp32 oracle: rel-L2 <=
1e-2 in bf16 and 1.3e-3 in fp16 (P is rounded to the input type, 2^-9 and 2^-12 relative, before the second contraction).
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
    "d64_items": (1, 12, 64, (8, 16, 24), (4, 8, 8), (4, 4, 4), torch.bfloat16),        # 288 items: two or more per CTA
    "d128_items": (1, 12, 128, (8, 16, 24), (4, 8, 8), (4, 4, 4), torch.bfloat16),
    "d128_items_ragged": (1, 10, 128, (8, 15, 23), (4, 7, 9), (4, 4, 4), torch.bfloat16),
    "blocks128_items": (1, 14, 128, (8, 16, 24), (4, 8, 16), (4, 4, 8), torch.bfloat16),  # 336 items of one block
    "blocks128_items_fp16": (1, 14, 128, (8, 15, 24), (4, 7, 16), (4, 4, 8), torch.float16),
}


@pytest.mark.parametrize("lists", ["short", "mixed"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_uneven_lists(name, lists):
    b, h, d, gq, gk, chunk, dt = SHAPES[name]
    wl = Workload(name, 9100 + sorted(SHAPES).index(name), b, h, d, gq, gk, chunk, 0.5, dt, "normal")
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


@pytest.mark.parametrize("d", [64, 128])
def test_growing_maximum_rescales(d):
    """Key blocks whose scores grow by far more than 2^8 from one to the next: every round moves the reference maximum."""
    gq, gk, chunk = (4, 8, 8), (4, 16, 16), (4, 4, 4)
    wl = Workload("grow", 9200 + d, 1, 2, d, gq, gk, chunk, 0.0, torch.bfloat16, "normal")
    q, k, v = make_qkv(wl)
    nq, nk = O.num_blocks(gq, chunk), O.num_blocks(gk, chunk)
    q = q.abs()
    order = torch.empty(gk[0] * gk[1] * gk[2])
    order[O.token_map(gk, chunk).long().flatten()] = torch.arange(nk).repeat_interleave(64).float()
    k = (k.abs() * 0.2 * (1.0 + order)[None, None, :, None]).to(k.dtype)
    idx = torch.arange(nk, dtype=torch.int32).expand(1, 2, nq, nk).contiguous()
    cnt = torch.full((1, 2, nq), nk, dtype=torch.int32)
    ref, _ = O.attention(q, k, v, gq, gk, chunk, chunk, idx, cnt)
    out = B.attn_fwd_bsa_varlen(q.cuda(), k.cuda(), v.cuda(), 1 / d ** 0.5, idx.cuda(), cnt.cuda(), gq, gk, chunk, chunk, impl=TC[d])
    assert rel_l2(out.float().cpu(), ref) <= TOL[torch.bfloat16]
