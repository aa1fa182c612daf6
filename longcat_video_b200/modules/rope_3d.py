"""q/k RMSNorm + 3-D rotary embedding in one CUDA pass: the step in front of the block-sparse attention.

Stands in for these lines of ``Attention.forward`` (``longcat_video/modules/attention.py:113-121``)::

    q, k = self.q_norm(q), self.k_norm(k)          # RMSNorm_FP32, longcat_video/modules/blocks.py:42-53
    q, k = self.rope_3d(q, k, grid_size=shape)     # longcat_video/modules/rope_3d.py:99-120

which run as six elementwise passes with fp32 temporaries.  ``qk_norm_rope`` reads the strided q and k views of the
fused qkv projection once and writes ``[B, H, S, D]`` outputs once.  All arithmetic is in liblcbsa.so
(``lcbsa_norm_rope_jobs``); PyTorch builds the small angle table and allocates the outputs.  There is no CPU path.
"""
from __future__ import annotations

import ctypes
from typing import NamedTuple, Optional, Sequence, Tuple

import torch

from .. import _lib as L

_TABLES = {}


def _angles(n: int, part: int, base: float, start: int = 0) -> torch.Tensor:
    """Angles of one axis for positions ``start .. start + n - 1``, ``[n, part]``: pair i of the part turns by
    ``pos / base**(2i/part)`` (rope_3d.py:62-84), repeated for both elements of the pair (rope_3d.py:113-115)."""
    inv = 1.0 / (base ** (torch.arange(0, part, 2)[: part // 2].float() / part))
    pos = torch.arange(start, start + n, dtype=torch.float32)
    return torch.repeat_interleave(pos[:, None] * inv[None, :], 2, dim=1)


def rope_table(grid_size: Sequence[int], head_dim: int, device, base: float = 10000.0,
               pos_offset: Sequence[int] = (0, 0, 0)) -> torch.Tensor:
    """The packed separable fp32 table ``lcbsa_norm_rope`` reads, cached per (grid, head_dim, base, offset, device).
    ``pos_offset`` is the (t, h, w) position of the grid's first token: a context-parallel rank that holds rows
    ``h0 ..`` and columns ``w0 ..`` of the frame (the split of rope_3d.py:91-95) passes ``(0, h0, w0)``.  Layout:
    ``cos_t [T, dt] sin_t [T, dt] cos_h [H, dh] sin_h [H, dh] cos_w [W, dh] sin_w [W, dh]`` with
    ``dh = 2 * (D // 6)`` and ``dt = D - 2 * dh`` -- the split of rope_3d.py:62-66.  The reference caches its
    ``[S, D]`` tables per grid the same way (rope_3d.py:86-97)."""
    T, H, W = (int(v) for v in grid_size)
    device = torch.device(device)
    off = tuple(int(v) for v in pos_offset)
    key = (T, H, W, int(head_dim), float(base), off, device)
    tab = _TABLES.get(key)
    if tab is None:
        dh = 2 * (head_dim // 6)
        dt = head_dim - 2 * dh
        parts = []
        for n, part, start in ((T, dt, off[0]), (H, dh, off[1]), (W, dh, off[2])):
            a = _angles(n, part, base, start)
            parts += [a.cos().reshape(-1), a.sin().reshape(-1)]
        tab = torch.cat(parts).contiguous()
        g = L.grid_desc((T, H, W), (1, 1, 1))
        want = L.lib().lcbsa_rope_table_floats(ctypes.byref(g), int(head_dim))
        if want != tab.numel():
            raise ValueError(f"rope table for grid {(T, H, W)}, head_dim {head_dim}: {tab.numel()} floats built, library expects {want}")
        tab = tab.to(device)
        _TABLES[key] = tab
    return tab


class RowJob(NamedTuple):
    """What ``run_row_jobs`` does to the rows of one ``[B, H, S, D]`` tensor (any B/H/S strides): RMSNorm times ``weight`` (None: off),
    the rotary embedding (``rope``), neither: a copy.  ``out_norm`` also keeps the rows as they are before the embedding."""
    x: torch.Tensor
    out: torch.Tensor
    weight: Optional[torch.Tensor]
    grid_size: Sequence[int]
    rope: bool = True
    t_offset: int = 0
    table_frames: Optional[int] = None
    pos_offset: Sequence[int] = (0, 0, 0)
    out_norm: Optional[torch.Tensor] = None


_NO_TENSOR = L.LcbsaTensor()


def run_row_jobs(jobs: Sequence[RowJob], eps: float = 1e-6, base: float = 10000.0) -> None:
    """One call for all jobs that share dtype, batch, heads and head_dim: for all there are, as a layer has them.  It is one launch
    where the jobs do not fill the chip, else a launch per job."""
    kinds = {}
    for j in jobs:
        if j.x.dim() != 4:
            raise ValueError("expected a [B, H, S, D] tensor")
        if j.out_norm is not None and (j.weight is None or not j.rope):
            raise ValueError("normalised rows are kept beside embedded ones: that takes a weight and the embedding")
        kinds.setdefault((j.x.dtype, j.x.device, j.x.shape[0], j.x.shape[1], j.x.shape[3]), []).append(j)
    for group in kinds.values():
        _launch_row_jobs(group, eps, base)


def _launch_row_jobs(jobs: Sequence[RowJob], eps: float, base: float) -> None:
    descs = (L.LcbsaRowJob * len(jobs))()
    keep = []  # weights and tables stay alive until the launch is queued
    for j, d in zip(jobs, descs):
        x, D = j.x, j.x.shape[3]
        if not L.abi_ok(x):
            x = x.contiguous()
        T = int(j.grid_size[0])
        frames = T + int(j.t_offset) if j.table_frames is None else int(j.table_frames)
        keep.append(x)
        if j.weight is not None:
            w = j.weight.to(device=x.device, dtype=x.dtype).contiguous()
            if w.numel() != D:
                raise ValueError(f"weight has {w.numel()} elements, head_dim is {D}")
            keep.append(w)
            d.weight = w.data_ptr()
        if j.rope:
            tab = rope_table((frames, j.grid_size[1], j.grid_size[2]), D, x.device, base, j.pos_offset)
            keep.append(tab)
            d.rope_tab = tab.data_ptr()
        d.x, d.out = L.tensor_desc(x), L.tensor_desc(j.out)
        d.out_norm = _NO_TENSOR if j.out_norm is None else L.tensor_desc(j.out_norm)
        d.grid, d.table_T, d.t_offset = L.grid_plan(j.grid_size, (1, 1, 1))[0], frames, int(j.t_offset)
    dev = jobs[0].x.device
    with L.on_device(dev):
        L.check(L.lib().lcbsa_norm_rope_jobs(descs, len(jobs), float(eps), L.current_stream(dev)))


def norm_rope(x: torch.Tensor, weight: Optional[torch.Tensor], grid_size: Sequence[int], eps: float = 1e-6, base: float = 10000.0,
              out: Optional[torch.Tensor] = None, rope: bool = True, t_offset: int = 0, table_frames: Optional[int] = None,
              pos_offset: Sequence[int] = (0, 0, 0)) -> torch.Tensor:
    """RMSNorm(x) * weight, then the 3-D rotary embedding, for one ``[B, H, S, D]`` tensor (any B/H/S strides).

    ``weight=None`` skips the normalisation and ``rope=False`` the embedding.  ``t_offset`` places the tensor's first
    frame at frame ``t_offset`` of a table of ``table_frames`` frames (default ``T + t_offset``): the new tokens behind
    cached frames (attention.py:165-169)."""
    if x.dim() != 4:
        raise ValueError("expected a [B, H, S, D] tensor")
    if weight is None and not rope:
        raise ValueError("neither normalisation nor rotary embedding requested")
    if out is None:
        out = torch.empty(x.shape, dtype=x.dtype, device=x.device)
    run_row_jobs([RowJob(x, out, weight, grid_size, rope, t_offset, table_frames, pos_offset)], eps, base)
    return out


def rms_norm(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-6, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``RMSNorm_FP32`` alone (blocks.py:42-53) on ``[B, H, S, D]``: what ``return_kv`` caches (attention.py:118-119)."""
    return norm_rope(x, weight, (x.shape[2], 1, 1), eps, out=out, rope=False)


def qk_norm_rope(q: torch.Tensor, k: torch.Tensor, q_weight: torch.Tensor, k_weight: torch.Tensor, grid_size: Sequence[int],
                 eps: float = 1e-6, base: float = 10000.0) -> Tuple[torch.Tensor, torch.Tensor]:
    """``rope_3d(q_norm(q), k_norm(k), grid_size)`` of attention.py:113-121 in one call (see ``run_row_jobs``)."""
    q_out, k_out = torch.empty(q.shape, dtype=q.dtype, device=q.device), torch.empty(k.shape, dtype=k.dtype, device=k.device)
    run_row_jobs([RowJob(q, q_out, q_weight, grid_size), RowJob(k, k_out, k_weight, grid_size)], eps, base)
    return q_out, k_out


def kv_cache_row_jobs(q: torch.Tensor, k: torch.Tensor, q_weight: torch.Tensor, k_weight: torch.Tensor, k_cache: torch.Tensor,
                      grid_size: Sequence[int], num_cond_latents: int) -> Tuple[torch.Tensor, torch.Tensor, list]:
    """Outputs and row jobs of ``qk_norm_rope_with_kv_cache``."""
    T, Hh, W = (int(v) for v in grid_size)
    nc = int(num_cond_latents)
    B, H, N, D = q.shape
    sc = nc * Hh * W
    if k_cache.shape[0] == 1 and B > 1:  # attention.py:160-162
        k_cache = k_cache.expand(B, -1, -1, -1)
    assert k_cache.shape[2] == sc and N == T * Hh * W
    k_full = torch.empty(B, H, sc + N, D, dtype=k.dtype, device=k.device)
    q_out = torch.empty(B, H, N, D, dtype=q.dtype, device=q.device)
    jobs = [RowJob(k_cache, k_full[:, :, :sc], None, (nc, Hh, W), table_frames=T + nc),
            RowJob(k, k_full[:, :, sc:], k_weight, grid_size, t_offset=nc), RowJob(q, q_out, q_weight, grid_size, t_offset=nc)]
    return q_out, k_full, jobs


def qk_norm_rope_with_kv_cache(q: torch.Tensor, k: torch.Tensor, q_weight: torch.Tensor, k_weight: torch.Tensor, k_cache: torch.Tensor,
                               grid_size: Sequence[int], num_cond_latents: int, eps: float = 1e-6, base: float = 10000.0
                               ) -> Tuple[torch.Tensor, torch.Tensor]:
    """The q / k part of ``forward_with_kv_cache`` (attention.py:156-171): returns q ``[B,H,N,D]`` and
    ``k_full [B,H,(NC+T)HW,D]``.  The reference concatenates the cache and the new keys, pads q in front with an empty
    tensor of the cache's size, embeds both over ``(T + NC, H, W)`` and cuts q's tail off again; here the cached keys
    are embedded into the head of ``k_full``, the new keys are normalised and embedded into its tail, and q is
    normalised and embedded at frame offset NC: one call, no padding and no concatenation."""
    q_out, k_full, jobs = kv_cache_row_jobs(q, k, q_weight, k_weight, k_cache, grid_size, num_cond_latents)
    run_row_jobs(jobs, eps, base)
    return q_out, k_full
