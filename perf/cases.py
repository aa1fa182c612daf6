"""The work this library is measured on: block-sparse attention calls as the LongCat-Video DiT makes them.

Every case goes through a public entry point -- ``flash_attn_bsa_3d`` (forward, and forward + backward through autograd)
or the layer bodies of ``longcat_video_b200.modules`` -- at a size of this repository's benchmark configurations and
tests, or a generic one.  ``listed()`` names them, ``draw()`` gives more of the same ranges, ``prepare()`` makes what a
caller has in hand (on the GPU, from the seed alone), ``run()`` is one pass.

A case is a dict of plain values:

  op        "attention": flash_attn_bsa_3d    "train": the same plus its gradients
            "layer": self_attention on views of a fused qkv projection    "layer_kv": self_attention_with_kv_cache
  T, H, W   latent grid of the queries        Tk: frames of the keys (attention; H and W are shared)
  cond      conditioning frames (layer: attend among themselves; layer_kv: cached)
  ct/ch/cw  3-D block of queries and keys     batch, heads, head_dim, dtype
  sparsity  share of key blocks left out      cdf: cdf_threshold, or 0 for none
"""
import math

import torch

from longcat_video_b200.block_sparse_attention.bsa_interface import flash_attn_bsa_3d
from longcat_video_b200.modules import self_attention, self_attention_with_kv_cache

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(op, grid, heads, block=(4, 4, 4), sparsity=0.9375, cdf=0.0, batch=1, head_dim=128, dtype="bf16", frames_k=0, cond=0):
    T, H, W = grid
    return {"op": op, "T": T, "H": H, "W": W, "Tk": frames_k or T, "cond": cond, "ct": block[0], "ch": block[1], "cw": block[2],
            "batch": batch, "heads": heads, "head_dim": head_dim, "dtype": dtype, "sparsity": sparsity, "cdf": cdf}


def listed():
    cases = {
        # the smallest call: a few blocks of two heads, where launches and the host path are the time (smoke-test shape)
        "attn_smallest": _case("attention", (8, 8, 12), 2, sparsity=0.75),
        # a low-resolution preview of a small model: head_dim 64 in fp16, batch 2 (guided and unguided together)
        "attn_preview_d64_fp16": _case("attention", (12, 16, 24), 16, sparsity=0.75, batch=2, head_dim=64, dtype="fp16"),
        # one self-attention of the DiT at 480p x 93 frames, all 32 heads, the model's own block and sparsity
        "attn_480p": _case("attention", (24, 32, 52), 32),
        # the refine stage at 720p x 93 frames: the layer most of a generation's time goes into
        "attn_720p": _case("attention", (24, 48, 80), 32),
        # the literal 720p latent (45 rows): partial edge blocks through the ragged extension
        "attn_720p_ragged": _case("attention", (24, 45, 80), 32),
        # every parameter of flash_attn_bsa_3d at its default: 128-token blocks, sparsity 0.875; the largest call
        "attn_720p_defaults": _case("attention", (24, 48, 80), 32, block=(4, 4, 8), sparsity=0.875),
        # video continuation at 720p: the generated half of the frames attends to all frames, heads of one of two ranks
        "attn_720p_continuation": _case("attention", (12, 48, 80), 16, frames_k=24, sparsity=0.875),
        # the cdf_threshold option together with a minimum share of blocks, 480p, heads of one of four ranks
        "attn_480p_cdf": _case("attention", (24, 32, 52), 8, cdf=0.3),
        # the layer body of image-to-video / continuation: fused qkv in, RMSNorm + rotary, cond / noise split
        "layer_480p_cond": _case("layer", (24, 32, 52), 32, cond=4),
        # the same layer with the conditioning frames' keys and values cached: 12 new frames behind 12 cached ones
        "layer_480p_kv_cache": _case("layer_kv", (12, 32, 52), 32, cond=12),
        # a training step's attention, forward and gradients, with the model's 64-token blocks
        "train_480p": _case("train", (24, 32, 52), 8),
        # the same with the default 128-token blocks and sparsity
        "train_480p_defaults": _case("train", (24, 32, 56), 8, block=(4, 4, 8), sparsity=0.875),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def draw(rng):
    """One more case: sizes log-uniform over the listed ranges, every third one ragged (block edges in mid-block)."""
    limit = 0.8 * max(_cost(c) for c in listed())
    while True:
        op = rng.choice(["attention"] * 5 + ["train"] * 3 + ["layer", "layer_kv"])
        block = rng.choice([(4, 4, 4), (4, 4, 4), (4, 4, 8), (2, 4, 8)] if op in ("attention", "train") else [(4, 4, 4), (4, 4, 8)])
        ragged = op in ("attention", "train") and rng.random() < 1 / 3

        def axis(lo, hi, step):
            n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
            return n if ragged else max(step, n // step * step)

        T, H, W = axis(4, 24, block[0]), axis(8, 48, block[1]), axis(12, 80, block[2])
        heads = int(round(math.exp(rng.uniform(0.0, math.log(32)))))
        case = _case(op, (T, H, W), heads, block, rng.choice([0.5, 0.75, 0.875, 0.9375, 0.96875]))
        case["dtype"] = rng.choice(["bf16", "bf16", "fp16"])
        if op == "layer":
            case["cond"] = rng.choice([0, block[0]]) if T > block[0] else 0
        elif op == "layer_kv":
            case["cond"] = block[0] * rng.randint(1, 3)
        elif op == "attention":
            case["head_dim"] = rng.choice([128, 128, 128, 64])
            case["batch"] = rng.choice([1, 1, 2])
            if rng.random() < 0.25:
                case["Tk"] = T + block[0] * rng.randint(1, 3)
            elif rng.random() < 0.2:
                case["cdf"] = round(rng.uniform(0.1, 0.4), 2)
        if _cost(case) <= limit and all(_selected(case, _blocks(case, f)) > 0 for f in (case["cond"] or case["T"], _frames_k(case))):
            return case


def _frames_k(case):
    return case["T"] + case["cond"] if case["op"] == "layer_kv" else case["Tk"]


def _blocks(case, frames):
    return -(-frames // case["ct"]) * -(-case["H"] // case["ch"]) * -(-case["W"] // case["cw"])


def _selected(case, n_k):
    """Key blocks per query block.  With cdf_threshold the count depends on the data; on these inputs at 480p it is 6.7 %
    of the blocks at 0.2, 9.2 % at 0.3 and 13.6 % at 0.4 when that is above the floor: about the threshold squared."""
    n = int((1.0 - case["sparsity"]) * n_k)
    return max(n, int(case["cdf"] ** 2 * n_k))


def _attention_flops(case):
    per_frame = case["H"] * case["W"]
    Tk = _frames_k(case)
    n_k = _blocks(case, Tk)
    keys = _selected(case, n_k) / n_k * Tk * per_frame  # present tokens only: edge blocks of ragged grids are partial
    scores = 2.0 * _blocks(case, case["T"]) * n_k * case["head_dim"]
    heads = case["batch"] * case["heads"]
    if case["op"] == "layer" and case["cond"]:
        nc = case["cond"]
        rest = 1.0 - nc / case["T"]
        n_c = _blocks(case, nc)
        keys = keys * rest + _selected(case, n_c) / n_c * nc * per_frame * (1.0 - rest)
    return heads * (4.0 * case["T"] * per_frame * keys * case["head_dim"] + scores)


def _cost(case):
    """Relative cost for draw(): shapes outside the 128-wide head and whole 64/128-token blocks run at a fraction of the rate."""
    f = _attention_flops(case) * (3.5 if case["op"] == "train" else 1.0)
    ragged = case["T"] % case["ct"] or case["H"] % case["ch"] or case["W"] % case["cw"]
    if case["head_dim"] != 128 or (case["op"] == "train" and ragged):
        f *= 8.0
    return f * (3.0 if case["cdf"] else 1.0)


def _spatial(case, frames, gen, rank=4):
    """A smooth function of the token's position, [tokens, rank]: what makes some blocks matter more than others."""
    H, W = case["H"], case["W"]
    dev = gen.device
    t = (torch.arange(frames, device=dev) / frames).view(-1, 1, 1).expand(frames, H, W).reshape(-1)
    h = (torch.arange(H, device=dev) / H).view(1, -1, 1).expand(frames, H, W).reshape(-1)
    w = (torch.arange(W, device=dev) / W).view(1, 1, -1).expand(frames, H, W).reshape(-1)
    freq = torch.randint(0, 4, (3, rank), generator=gen, device=dev).float()
    phase = torch.rand(rank, generator=gen, device=dev) * (2 * math.pi)
    return torch.cos(2 * math.pi * (t[:, None] * freq[0] + h[:, None] * freq[1] + w[:, None] * freq[2]) + phase)


def _normal(gen, dtype, *shape):
    return torch.randn(shape, generator=gen, device=gen.device, dtype=torch.float32).to(dtype)


def prepare(case, seed):
    """Queries and keys as they leave q_norm / k_norm (unit variance) plus a position-dependent part, so that the block
    lists are neither uniform nor the same for all queries; values of unit variance."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    B, h, D = case["batch"], case["heads"], case["head_dim"]
    T, H, W = case["T"], case["H"], case["W"]
    S = T * H * W
    params = dict(sparsity=case["sparsity"], cdf_threshold=case["cdf"] or None,
                  chunk_3d_shape_q=[case["ct"], case["ch"], case["cw"]], chunk_3d_shape_k=[case["ct"], case["ch"], case["cw"]])
    state = {"op": case["op"], "shape": (T, H, W), "cond": case["cond"], "params": params}
    if case["op"] in ("layer", "layer_kv"):
        qkv = _normal(gen, dt, B, S, 3, h, D)  # the fused projection; its views go in as they are
        mix = (torch.randn(4, h, D, generator=gen, device=gen.device) * 0.5).to(dt)
        qkv[:, :, :2] += torch.einsum("sr,rhd->shd", _spatial(case, T, gen).to(dt), mix)[None, :, None]
        state["q"], state["k"], state["v"] = qkv.permute(2, 0, 3, 1, 4).unbind(0)
        state["wq"], state["wk"] = (1.0 + 0.2 * torch.randn(2, D, generator=gen, device=gen.device)).to(dt).unbind(0)
        if case["op"] == "layer_kv":
            state["cache"] = (_normal(gen, dt, B, h, case["cond"] * H * W, D), _normal(gen, dt, B, h, case["cond"] * H * W, D))
        return state
    Tk = case["Tk"]
    mix = (torch.randn(h, 4, D, generator=gen, device=gen.device) * 0.35).to(dt)
    pos = _spatial(case, max(T, Tk), gen).to(dt)
    q = _normal(gen, dt, B, h, S, D) + torch.matmul(pos[:S], mix)
    k = _normal(gen, dt, B, h, Tk * H * W, D) + torch.matmul(pos[:Tk * H * W], mix)
    v = _normal(gen, dt, B, h, Tk * H * W, D)
    if any(n % c for n, c in ((T, case["ct"]), (Tk, case["ct"]), (H, case["ch"]), (W, case["cw"]))):
        params["allow_ragged"] = True
    state.update(q=q, k=k, v=v, shape_k=(Tk, H, W))
    if case["op"] == "train":
        for n in "qkv":
            state[n].requires_grad_(True)
        state["grad"] = _normal(gen, dt, B, h, S, D)
    return state


def run(state):
    q, k, v = state["q"], state["k"], state["v"]
    if state["op"] == "layer":
        if state["cond"]:  # the step that also fills the cache for what follows
            x, kv = self_attention(q, k, v, state["wq"], state["wk"], state["shape"], state["params"], num_cond_latents=state["cond"],
                                   return_kv=True)
            return (x, *kv)
        return self_attention(q, k, v, state["wq"], state["wk"], state["shape"], state["params"])
    if state["op"] == "layer_kv":
        return self_attention_with_kv_cache(q, k, v, state["wq"], state["wk"], state["shape"], state["cache"], state["params"],
                                            state["cond"])
    out = flash_attn_bsa_3d(q, k, v, state["shape"], state["shape_k"], **state["params"])
    if state["op"] == "train":
        return (out, *torch.autograd.grad(out, (q, k, v), state["grad"]))
    return out


def work(case):
    """Inputs read once, outputs written once; the contractions over the selected blocks (two forward, five backward)
    and the block scores."""
    H, W = case["H"], case["W"]
    rows = case["batch"] * case["heads"] * case["head_dim"] * 2
    n_q, n_k = case["T"] * H * W, _frames_k(case) * H * W
    tensors = 2 * n_q + 2 * n_k  # q, out; k, v
    if case["op"] == "train":
        tensors += 2 * n_q + 2 * n_k  # the result's gradient in; dq, dk, dv out
    if case["op"] == "layer" and case["cond"]:
        tensors += 2 * n_k  # the cached k and v
    flops = _attention_flops(case)
    return {"bytes": float(rows * tensors), "flops": flops * (3.5 if case["op"] == "train" else 1.0)}


def tolerance(case):
    """bf16 and fp16 results with fp32 sums: the probabilities (and, backward, their gradients) are rounded to the input
    type before the second contraction.  Measured against the same path in float64 (2 heads of an 8x16x24 grid): forward
    2.3e-3 in bf16 and 2.9e-4 in fp16, gradients 2.8e-3 and 3.5e-4; stated at about four times that."""
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 1.3e-3}
