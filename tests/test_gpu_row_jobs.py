"""Several row jobs in one call (``lcbsa_norm_rope_jobs``) against the same jobs one by one, bit for bit: the launch that serves all kinds
and the launches per job, remainders in tokens and heads, batch strides of 0, rows that are not numbers."""
import pytest
import torch

from longcat_video_b200.modules import rope_3d as R
from longcat_video_b200.modules.attention import self_attention

pytestmark = pytest.mark.gpu


def _bits(t):
    return t.contiguous().view(torch.int16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B, H, D, grid", [
    (1, 3, 128, (2, 4, 4)),      # one block of 32 tokens
    (2, 17, 64, (3, 5, 7)),      # remainders in tokens and heads
    (2, 2, 128, (1, 1, 33)),
    (1, 33, 128, (8, 33, 41)),   # enough CTAs for a launch per job
    (3, 18, 64, (6, 33, 41)),
])
def test_jobs_together_equal_jobs_alone(dtype, B, H, D, grid):
    S = grid[0] * grid[1] * grid[2]
    gen = torch.Generator(device="cuda").manual_seed(S + H)
    qkv = (torch.randn(B, S, 3, H, D, generator=gen, device="cuda") * 1.5).to(dtype)
    q, k, v = qkv.permute(2, 0, 3, 1, 4).unbind(0)
    v[0, 0, 0, 0], v[0, 0, S - 1, D - 1], v[0, H - 1, 0, 1] = float("nan"), float("inf"), -0.0
    wq, wk = (1.0 + 0.2 * torch.randn(2, D, generator=gen, device="cuda")).to(dtype).unbind(0)
    cache = (torch.randn(1, H, S, D, generator=gen, device="cuda")).to(dtype).expand(B, -1, -1, -1)
    new = lambda: torch.empty(B, H, S, D, dtype=dtype, device="cuda")  # noqa: E731
    both = torch.empty(B, H, 2 * S, D, dtype=dtype, device="cuda")
    outs = [new(), new(), new(), torch.empty_like(v), new()]
    R.run_row_jobs([R.RowJob(q, outs[0], wq, grid), R.RowJob(k, outs[1], wk, grid, out_norm=outs[2]), R.RowJob(v, outs[3], None, grid, rope=False),
                    R.RowJob(cache, both[:, :, :S], None, grid), R.RowJob(k, both[:, :, S:], wk, grid, t_offset=3), R.RowJob(k, outs[4], wk, grid, rope=False)])
    assert outs[3].stride() == v.clone().stride()
    want = [R.norm_rope(q, wq, grid), R.norm_rope(k, wk, grid), R.rms_norm(k, wk), v, R.rms_norm(k, wk)]
    for got, ref in zip(outs, want):
        assert torch.equal(_bits(got), _bits(ref))
    assert torch.equal(_bits(both[:, :, :S]), _bits(R.norm_rope(cache, None, grid)))
    assert torch.equal(_bits(both[:, :, S:]), _bits(R.norm_rope(k, wk, grid, t_offset=3)))


def test_copies_that_differentiation_sees_stay_with_torch():
    """v that requires grad: the cached copy is part of the graph, as it was."""
    grid, params = (4, 8, 8), dict(sparsity=0.5, chunk_3d_shape_q=[4, 4, 4], chunk_3d_shape_k=[4, 4, 4])
    S = grid[0] * grid[1] * grid[2]
    q, k, v = (torch.randn(1, 2, S, 128, device="cuda").bfloat16() for _ in range(3))
    w = torch.ones(128, device="cuda").bfloat16()
    x, (kc, vc) = self_attention(q, k, v.requires_grad_(True), w, w, grid, params, return_kv=True)
    gx, = torch.autograd.grad(x.float().sum() + 2 * vc.float().sum(), v)
    x2, = torch.autograd.grad(self_attention(q, k, v, w, w, grid, params).float().sum(), v)
    assert vc.requires_grad and not kc.requires_grad
    assert torch.allclose(gx.float(), x2.float() + 2.0, atol=2.0 ** -5)
