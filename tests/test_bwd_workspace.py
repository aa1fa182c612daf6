"""Size of the backward's workspace (host arithmetic, no GPU)."""
import ctypes

import pytest

from longcat_video_b200 import _lib as L


def _bytes(grid_q, grid_k, block, heads, cap):
    S = grid_q[0] * grid_q[1] * grid_q[2]
    q = L.LcbsaTensor(0, L.LCBSA_BF16, 0, (ctypes.c_int64 * 4)(1, heads, S, 128), (ctypes.c_int64 * 4)(heads * S * 128, S * 128, 128, 1))
    gq, gk = L.grid_desc(grid_q, block), L.grid_desc(grid_k, block)
    return L.lib().lcbsa_attn_bwd_workspace_bytes(ctypes.byref(q), ctypes.byref(gq), ctypes.byref(gk), cap)


@pytest.mark.parametrize("ragged, block", [((24, 45, 80), (4, 4, 4)), ((5, 9, 13), (4, 4, 4)), ((3, 5, 9), (2, 4, 8)), ((1, 1, 1), (4, 4, 4))])
def test_ragged_grids_have_room_for_every_slot(ragged, block):
    """The passes lay (lse, delta) out per slot of every query block, and a ragged grid has more slots than tokens.  A ragged
    grid and the whole grid around it have the same blocks, so their workspaces differ by the 4 bytes of delta per token alone."""
    heads, cap = 8, 3
    whole = tuple(-(-n // c) * c for n, c in zip(ragged, block))
    tokens = lambda g: g[0] * g[1] * g[2]  # noqa: E731
    delta = 4 * heads * (tokens(whole) - tokens(ragged))
    assert _bytes(ragged, ragged, block, heads, cap) >= _bytes(whole, whole, block, heads, cap) - delta - 256
