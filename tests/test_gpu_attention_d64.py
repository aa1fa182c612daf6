"""head_dim 64: precision against float64, which kernel a call takes, and the calls that stay on the warp-level kernel.

The kernel is read off the nodes of a captured graph: a forced ``ATTN_TC`` refuses head_dim 64, so the tcgen05 form is only
reached by ``ATTN_AUTO``, and a comparison with ``ATTN_MMA`` alone would also pass if that chose the warp-level kernel.
"""
import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B
from longcat_video_b200.synthetic import Workload, make_qkv
from oracle import bsa_oracle as O
from tests.golden.cases import CASES
from tests.helpers import kernels_of_capture, load_golden, rel_l2
from tests.test_gpu_attention_items import LONG, SHAPES

pytestmark = pytest.mark.gpu


def _dense(q, k, v, gq, gk, chunk, idx, cnt):
    """float64 softmax over the keys of every list, on the device."""
    tq, tk = O.token_map(gq, chunk).cuda(), O.token_map(gk, chunk).cuda()
    out = torch.zeros(q.shape, dtype=torch.float64, device="cuda")
    for b in range(q.shape[0]):
        for h in range(q.shape[1]):
            for n in range(tq.shape[0]):
                rows = tq[n][tq[n] >= 0]
                keys = tk[idx[b, h, n, : int(cnt[b, h, n])].long()].flatten()
                keys = keys[keys >= 0]
                s = (q[b, h, rows].double() @ k[b, h, keys].double().T) * q.shape[-1] ** -0.5
                out[b, h, rows] = torch.softmax(s, -1) @ v[b, h, keys].double()
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["normal", "scaled_lowrank"])
@pytest.mark.parametrize("gq,gk,chunk,sparsity", [
    ((12, 16, 24), (12, 16, 24), (4, 4, 4), 0.75),
    ((4, 16, 16), (8, 16, 16), (4, 4, 4), 0.5),
    ((8, 15, 22), (8, 15, 22), (2, 4, 8), 0.875),
    ((8, 16, 24), (8, 16, 24), (4, 4, 4), 0.96875),
])
def test_no_further_from_float64_than_the_warp_level_kernel(gq, gk, chunk, sparsity, kind, dtype):
    """Both round P to the input type; where a row's largest probability is exactly 1 its rounding does not count, so the
    reference has to be the running maximum.  The errors are norms over 130 000 elements and more, whose spread is
    1 / sqrt(2 n) < 0.2 %: 1 % is allowed for it."""
    wl = Workload("d64", 9400, 1, 2, 64, gq, gk, chunk, sparsity, dtype, kind)
    q, k, v = (t.cuda() for t in make_qkv(wl))
    idx, cnt = B.get_select_indices(q, k, gq, gk, sparsity, None, chunk, chunk)
    want = _dense(q, k, v, gq, gk, chunk, idx, cnt)
    err = {}
    for impl in (L.ATTN_AUTO, L.ATTN_MMA):
        got = B.attn_fwd_bsa_varlen(q, k, v, 64 ** -0.5, idx, cnt, gq, gk, chunk, chunk, impl=impl).double()
        err[impl] = float((got - want).norm() / want.norm())
    L.check(L.lib().lcbsa_check_device_status())
    print(f"D64 {gq} {sparsity} {kind} {dtype}: AUTO {err[L.ATTN_AUTO]:.4e} warp-level {err[L.ATTN_MMA]:.4e}")
    assert err[L.ATTN_AUTO] <= 1.01 * err[L.ATTN_MMA]


def _call(gq, gk, chunk, dtype, d=64):
    g = torch.Generator().manual_seed(0)
    q, k, v = (torch.randn(1, 2, s[0] * s[1] * s[2], d, generator=g).to(dtype).cuda() for s in (gq, gk, gk))
    nq, nk = O.num_blocks(gq, chunk), O.num_blocks(gk, chunk)
    idx = torch.arange(nk, dtype=torch.int32).expand(1, 2, nq, nk).contiguous().cuda()
    cnt = torch.full((1, 2, nq), nk, dtype=torch.int32).cuda()
    return lambda impl, scale=d ** -0.5: B.attn_fwd_bsa_varlen(q, k, v, scale, idx, cnt, gq, gk, chunk, chunk, impl=impl)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_a_negative_scale_stays_on_the_warp_level_kernel(dtype):
    """Bit for bit what the warp-level kernel gives, at scales where an fp16 P comes near its largest value."""
    call = _call((4, 8, 8), (4, 8, 16), (4, 4, 4), dtype)
    for scale in (-0.125, -0.25):
        assert torch.equal(call(L.ATTN_AUTO, scale).view(torch.int16), call(L.ATTN_MMA, scale).view(torch.int16))
    L.check(L.lib().lcbsa_check_device_status())
    assert any("attn_mma_kernel" in k for k in kernels_of_capture(lambda: call(L.ATTN_AUTO, -0.125)))


FORMS = {n: c for n, c in {**SHAPES, **LONG}.items() if c[2] == 64}


@pytest.mark.parametrize("name", sorted(FORMS))
def test_64_token_blocks_take_the_tcgen05_kernel(name):
    """The shapes that the head_dim 64 tests of this kernel use reach it: dtype, ragged form and head_dim of the instantiation."""
    b, h, d, gq, gk, chunk, dt = FORMS[name]
    ragged = any(n % c for n, c in zip(gk, chunk))
    names = kernels_of_capture(lambda c=_call(gq, gk, chunk, dt, d): c(L.ATTN_AUTO))
    want = f"attn_tc_kernelILb{int(dt == torch.bfloat16)}ELb{int(ragged)}ELi64E"
    assert any(want in k for k in names) and not any("attn_mma_kernel" in k for k in names), names


def test_128_token_blocks_stay_on_the_warp_level_kernel():
    names = kernels_of_capture(lambda c=_call((4, 8, 16), (4, 8, 16), (4, 4, 8), torch.bfloat16): c(L.ATTN_AUTO))
    assert any("attn_mma_kernel" in k for k in names) and not any("attn_tc" in k for k in names), names


def test_golden_case_on_the_kernel_that_serves_it():
    """Lists and result of the reference's own functions at head_dim 64 (fixture fp16_d64), through the dispatch of a user's call."""
    wl, _ = CASES["fp16_d64"]
    gold = load_golden("fp16_d64")
    q, k, v = make_qkv(wl)
    idx = torch.sort(torch.from_numpy(gold["idx"].astype("int32")), dim=-1).values.contiguous().cuda()
    cnt = torch.from_numpy(gold["lens"].astype("int32")).cuda()
    ref = torch.from_numpy(gold["attn"])
    q, k, v = q.cuda(), k.cuda(), v.cuda()

    def call():
        return B.attn_fwd_bsa_varlen(q, k, v, wl.head_dim ** -0.5, idx, cnt, wl.grid_q, wl.grid_k, wl.chunk, wl.chunk)

    names = kernels_of_capture(call)
    assert any("attn_tc_kernel" in n for n in names), names
    out = call().float().cpu()
    L.check(L.lib().lcbsa_check_device_status())
    assert rel_l2(out, ref) <= 1.3e-3  # fp16: P is rounded to 2^-12 relative
