"""Device memory that a call of the operator holds beside its inputs and its result."""
import ctypes

import pytest
import torch

from longcat_video_b200 import _lib as L
from longcat_video_b200.block_sparse_attention import bsa_interface as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid, heads, large", [((12, 32, 52), 32, True), ((8, 8, 12), 2, False)])
def test_a_large_workspace_of_the_selection_is_gone_when_the_output_is_allocated(grid, heads, large):
    chunk, sparsity, D = (4, 4, 4), 0.9375, 128
    S = grid[0] * grid[1] * grid[2]
    g, n = L.grid_plan(grid, chunk)
    q, k, v = (torch.randn(1, heads, S, D, device="cuda").bfloat16() for _ in range(3))
    d = L.tensor_desc(q)
    ws = L.lib().lcbsa_select_workspace_bytes_fast(ctypes.byref(d), ctypes.byref(d), ctypes.byref(g), ctypes.byref(g))
    assert (ws > B._SHARED_WORKSPACE_BYTES) == large
    lists = heads * n * 4 * (B.num_selected(sparsity, n) + 1)
    out = q.numel() * 2
    args = (q, k, v, grid, grid)
    params = dict(sparsity=sparsity, chunk_3d_shape_q=list(chunk), chunk_3d_shape_k=list(chunk))
    B.flash_attn_bsa_3d(*args, **params)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    B.flash_attn_bsa_3d(*args, **params)
    peak = torch.cuda.max_memory_allocated() - before
    rounding = 4096  # the allocator's units of 512 bytes, the parts' of 256
    assert peak <= lists + (max(ws, out) if large else ws + out) + rounding
