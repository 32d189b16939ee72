"""Workloads of the sparse-attention path: what a video DiT has this package do, from a single small
layer to the largest shipped one, through the public entry points.

A case is one call (or one short sequence of operator calls) of a kind:

  layer      sparse_attention_layer on Q, K, V of one self-attention layer, clustering included
  joint      the same with dense text tokens behind the video tokens (HunyuanVideo attention)
  reuse      a denoising step that keeps the clustering of an earlier one: map, permute, attention
  operators  the reference's operator names one by one: cluster, permute, map, attend, inverse permute
  wan        WanAttn_SAPAttn_Processor on hidden states: projections, norm, rotary embedding, layer, output
  hunyuan    Hunyuan_SAPAttn_Processor2_0 on a single-stream block (video tokens, then text tokens)
  ear        sparse_attention_layer with error-aware routing
  euclid     plain Euclidean k-means of one side (the use_svoo = False mode)

Tokens are the (t, h, w) latent grid in frame-major order.  Q, K, V and hidden states are a smooth
low-frequency field over the grid plus noise (so that clusters exist), RMS-normalised and rotated
with a 3-D rotary embedding where the model does so.  bf16 is the only element type of the kernels.
"""
from __future__ import annotations

import math
import os
import tempfile

import torch

from svoo_b200 import co_clustering, layer, permute, processor, sparsity, wan_dit

D = 128


# ------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------
def _case(name, kind, heads, grid, q, k, iters, lo, hi, text=0, prompt=0):
    """lo, hi: range of the per-head density budget (fraction of the key clusters a query cluster keeps)."""
    c = dict(kind=kind, heads=heads, t=grid[0], h=grid[1], w=grid[2], q=q, k=k, iters=iters, lo=lo, hi=hi, text=text,
             prompt=prompt)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest calls: four heads of 960 tokens, operator by operator (launches and host time) ...
        _case("operators-4x960", "operators", 4, (3, 16, 20), 12, 40, 2, 0.15, 0.15),
        # ... and a small layer with many iterations
        _case("layer-2x4096", "layer", 2, (4, 32, 32), 32, 128, 10, 0.2, 0.2),
        # the shipped cluster counts (256 / 1024, two iterations) on a ragged odd-sized video
        _case("layer-6x13727", "layer", 6, (7, 37, 53), 256, 1024, 2, 0.1, 0.1),
        # Wan2.1-1.3B at 480p, one layer
        _case("layer-12x32760", "layer", 12, (21, 30, 52), 100, 500, 5, 0.05, 0.30),
        # one GPU's heads of Wan2.1-14B at 720p when eight GPUs share the layer
        _case("layer-5x75600", "layer", 5, (21, 45, 80), 100, 500, 5, 0.05, 0.25),
        # Wan2.1-14B at 720p, one layer: the default benchmark
        _case("layer-40x75600", "layer", 40, (21, 45, 80), 100, 500, 5, 0.05, 0.25),
        # HunyuanVideo at 720p: joint attention with 256 text tokens
        _case("joint-24x118800", "joint", 24, (33, 45, 80), 128, 640, 5, 0.05, 0.20, 256, 256),
        # a denoising step that reuses the clustering
        _case("reuse-12x32760", "reuse", 12, (21, 30, 52), 100, 500, 0, 0.05, 0.30),
        # the attention of a Wan2.1-1.3B block as the DiT calls it, 49 frames at 480p
        _case("wan-12x20280", "wan", 12, (13, 30, 52), 100, 500, 5, 0.05, 0.30),
        # a HunyuanVideo single-stream block on a short odd-sized clip, shipped cluster counts, part of the prompt unused
        _case("hunyuan-24x8505", "hunyuan", 24, (9, 27, 35), 256, 1024, 2, 0.1, 0.1, 256, 203),
        # error-aware routing: block scores, budgeted selection, centroid keys for the pruned blocks
        _case("ear-12x32760", "ear", 12, (21, 30, 52), 100, 500, 5, 0.05, 0.25),
        # Euclidean k-means of the keys of one layer
        _case("euclid-12x32760", "euclid", 12, (21, 30, 52), 0, 500, 5, 0.0, 0.0),
    ]


def _pairs(c):
    """Query-key pairs that the attention cannot do without, summed over the heads, from the budgets alone."""
    n, s = c["t"] * c["h"] * c["w"], c["t"] * c["h"] * c["w"] + c["text"]
    rho = 0.5 * (c["lo"] + c["hi"]) * (2.0 if c["kind"] == "ear" else 1.0)
    pairs = rho * n * n + n * c["prompt"] + c["prompt"] * (n + c["prompt"]) + (c["text"] - c["prompt"]) ** 2
    if c["kind"] == "ear":
        pairs += n * c["k"]                                   # one centroid key per cluster
    return 0.0 if c["kind"] == "euclid" else c["heads"] * min(pairs, float(s) * s)


def _projection_flops(c):
    s = c["t"] * c["h"] * c["w"] + c["text"]
    return 8.0 * s * (c["heads"] * D) ** 2 if c["kind"] in ("wan", "hunyuan") else 0.0


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "joint", "reuse", "operators", "wan", "hunyuan", "ear", "euclid"])
    while True:
        grid = (rng.randint(2, 33), _log(rng, 12, 45), _log(rng, 16, 80))
        n = grid[0] * grid[1] * grid[2]
        heads = _log(rng, 1, 40)
        q, k = _log(rng, 12, 256), _log(rng, 40, 1024)
        if n < 960 or k > n // 8 or q > k:
            continue
        text = rng.choice([64, 256, 177]) if kind in ("joint", "hunyuan") else 0
        prompt = rng.randint(1, text) if text else 0
        lo = round(rng.uniform(0.05, 0.2), 3)
        hi = round(lo + rng.uniform(0.0, 0.1), 3)
        iters = 0 if kind == "reuse" else rng.randint(1, 10)
        c = _case("", kind, heads, grid, q, k, iters, lo, hi, text, prompt)
        w = work(c)
        # no dearer than the largest listed layer; the projections of a block count at their own rate
        if w["flops"] > 20e12 or _projection_flops(c) > 6e12 or heads * n > 2_900_000:
            continue
        return c


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _field(grid, width, gen, dev, waves=16):
    """[n, width] fp32: `waves` low-frequency cosines over the latent grid with random amplitudes, plus noise."""
    t, h, w = (torch.arange(g, device=dev, dtype=torch.float32) / g for g in grid)
    pos = torch.stack(torch.meshgrid(t, h, w, indexing="ij"), -1).reshape(-1, 3)
    freq = torch.randint(0, 4, (waves, 3), generator=gen, device=dev).float()
    freq[freq.sum(-1) == 0, 0] = 1.0
    phase = torch.rand(waves, generator=gen, device=dev) * (2 * math.pi)
    x = torch.cos(2 * math.pi * (pos @ freq.T) + phase) @ (torch.randn(waves, width, generator=gen, device=dev) / 4)
    return x.add_(torch.randn(x.shape, generator=gen, device=dev), alpha=0.5)


def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)


def _rotate(x, cos, sin):
    out = torch.empty_like(x)
    a, b, c, s = x[..., 0::2], x[..., 1::2], cos[..., 0::2], sin[..., 1::2]
    out[..., 0::2] = a * c - b * s
    out[..., 1::2] = a * s + b * c
    return out


def _qkv(c, gen, dev, which=3):
    """Q, K, V as [1, heads, tokens, 128] bf16, text tokens last."""
    grid = (c["t"], c["h"], c["w"])
    n, s = grid[0] * grid[1] * grid[2], grid[0] * grid[1] * grid[2] + c["text"]
    cos, sin = (r.reshape(n, D).to(dev) for r in wan_dit.rope_tables(grid))
    out = [torch.empty(1, c["heads"], s, D, dtype=torch.bfloat16, device=dev) for _ in range(which)]
    for head in range(c["heads"]):
        for i, dst in enumerate(out):
            x = _rms(_field(grid, D, gen, dev))
            dst[0, head, :n] = _rotate(x, cos, sin) if i < 2 else x
            if c["text"]:
                dst[0, head, n:] = _rms(torch.randn(c["text"], D, generator=gen, device=dev))
    return out


def _init_indices(c, gen, dev):
    n = c["t"] * c["h"] * c["w"]
    return (torch.randint(0, n, (c["heads"], max(c["q"], 1)), generator=gen, device=dev),
            torch.randint(0, n, (c["heads"], c["k"]), generator=gen, device=dev))


def _densities(c):
    """Per-head budgets spread over [lo, hi] in a fixed irregular order (the offline profile's table)."""
    return [round(c["lo"] + (c["hi"] - c["lo"]) * ((0.618034 * (i + 1)) % 1.0), 4) for i in range(c["heads"])]


def _attention_module(c, gen, dev):
    """The attention module of a DiT block: projections and weight-only RMS norms, random weights."""
    dim = c["heads"] * D
    attn = wan_dit.Attention(dim, c["heads"], 1e-6).to(device=dev, dtype=torch.bfloat16)
    if c["kind"] == "hunyuan":                                # norms over the 128 columns of a head
        attn.norm_q = wan_dit.RMSNormAcrossHeads(D, 1e-6).to(device=dev, dtype=torch.bfloat16)
        attn.norm_k = wan_dit.RMSNormAcrossHeads(D, 1e-6).to(device=dev, dtype=torch.bfloat16)
        attn.add_q_proj = None
    with torch.no_grad():
        for p in attn.parameters():
            if p.dim() == 2:
                p.copy_(torch.randn(p.shape, generator=gen, device=dev) / dim ** 0.5)
            elif p.numel() == dim and p is not attn.norm_q.weight and p is not attn.norm_k.weight:
                p.copy_(0.05 * torch.randn(p.shape, generator=gen, device=dev))
            else:
                p.copy_(1.0 + 0.1 * torch.randn(p.shape, generator=gen, device=dev))
    return attn


def _density_table(c):
    """The per-(step, layer, head) profile as the installer loads it."""
    fd, path = tempfile.mkstemp(suffix=".csv")
    with os.fdopen(fd, "w") as f:
        f.write("Step,Layer,Head,Sparsity\n")
        for i, d in enumerate(_densities(c)):
            f.write(f"1,0,{i},{d}\n")
    try:
        return sparsity.SparsityLookup(path)
    finally:
        os.unlink(path)


def _processor(c, indices):
    """A configured processor of layer 0 at step 1; the random initial tokens of a clustering come from the case's seed."""
    base = processor.WanAttn_SAPAttn_Processor if c["kind"] == "wan" else processor.Hunyuan_SAPAttn_Processor2_0
    cls = type(base.__name__, (base,), dict(
        num_frame=c["t"], frame_size=c["h"] * c["w"], context_length=c["text"], prompt_length=c["prompt"], num_layers=1,
        num_q_centroids=c["q"], num_k_centroids=c["k"], top_p_kmeans=0.0, min_kc_ratio=c["lo"], kmeans_iter_init=c["iters"],
        kmeans_iter_step=c["iters"], first_times_fp=float("inf"), sparsity_lookup=_density_table(c),
        use_dynamic_min_kc_ratio=True, draw_init_indices=lambda self, BH, N, device: indices))
    proc = cls(0)
    proc._step_from_callback = 1
    return proc


def prepare(case, seed):
    c, dev = case, torch.device("cuda")
    gen = torch.Generator(dev).manual_seed(seed)
    state = dict(case=c, indices=_init_indices(c, gen, dev), ratio=_densities(c))
    grid = (c["t"], c["h"], c["w"])
    if c["kind"] in ("wan", "hunyuan"):
        n, dim = grid[0] * grid[1] * grid[2], c["heads"] * D
        state["hidden"] = _field(grid, dim, gen, dev)[None].bfloat16()
        state["attn"] = _attention_module(c, gen, dev)
        state["proc"] = _processor(c, state["indices"])
        cos, sin = (r.to(dev) for r in wan_dit.rope_tables(grid))
        state["rotary"] = (cos, sin) if c["kind"] == "wan" else (cos.reshape(n, D), sin.reshape(n, D))
        if c["kind"] == "hunyuan":
            state["text"] = torch.randn(1, c["text"], dim, generator=gen, device=dev).bfloat16()
        return state
    if c["kind"] == "euclid":
        state["x"] = _qkv(c, gen, dev, which=1)[0][0]
        return state
    state["q"], state["k"], state["v"] = _qkv(c, gen, dev)
    if c["kind"] == "reuse":
        state["clustering"] = co_clustering.co_cluster(state["q"][0], state["k"][0], c["q"], c["k"], 2, init_indices=state["indices"])
    return state


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
@torch.no_grad()
def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "wan":
        return state["proc"](state["attn"], state["hidden"], rotary_emb=state["rotary"], timestep=500.0)
    if kind == "hunyuan":
        return state["proc"](state["attn"], state["hidden"], encoder_hidden_states=state["text"],
                             image_rotary_emb=state["rotary"], timestep=500.0)
    if kind == "euclid":
        labels, centroids, sizes, _ = co_clustering.batch_kmeans_Euclid(state["x"], c["k"], max_iters=c["iters"],
                                                                        init_indices=state["indices"][1])
        return labels, centroids, sizes
    q, k, v = state["q"], state["k"], state["v"]
    if kind == "operators":
        _, h, s, d = q.shape
        ql, qc, qs, kl, kc, ks = co_clustering.co_cluster_tokens(q[0], k[0], c["q"], c["k"], c["iters"],
                                                                 init_indices=state["indices"])
        qp, q_idx = permute.permute_tensor_by_labels_triton(q, ql[None], 2, num_clusters=c["q"])
        kp, k_idx = permute.permute_tensor_by_labels_triton(k, kl[None], 2, num_clusters=c["k"])
        vp, _ = permute.permute_tensor_by_labels_triton(v, None, 2, sorted_indices=k_idx)
        keep = co_clustering.identify_dynamic_map(qc[None], kc[None], qs[None], ks[None], 0.9, state["ratio"], state["ratio"])
        out = co_clustering.dynamic_block_sparse_fwd_flashinfer(qp, kp, vp, keep, qs[None], ks[None], is_cpu=False)
        return permute.apply_inverse_permutation_triton(out, q_idx, 2), ql, kl, keep
    ratio = state["ratio"]
    return layer.sparse_attention_layer(
        q, k, v, num_q_centroids=c["q"], num_k_centroids=c["k"], kmeans_iters=c["iters"], top_p=0.0 if kind == "ear" else 0.9,
        min_kc_ratio=ratio, max_kc_ratio=ratio, init_indices=state["indices"], clustering=state.get("clustering"),
        context_length=c["text"], prompt_length=c["prompt"] if c["text"] else None, ear_gamma=1.0 if kind == "ear" else None)


# ------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct implementations are apart
# ------------------------------------------------------------------------------------------
def work(case):
    """Flops: one [tokens, 128] x [128, clusters] product per side and iteration, the attention over
    the budgeted pairs, the block's projections.  Bytes: the inputs once, the outputs once."""
    c = case
    h, n = c["heads"], c["t"] * c["h"] * c["w"]
    s = n + c["text"]
    if c["kind"] == "euclid":
        return dict(bytes=h * n * (2.0 * D + 8) + h * c["k"] * (2.0 * D + 4), flops=c["iters"] * 2.0 * h * n * D * c["k"])
    flops = c["iters"] * 2.0 * h * n * D * (c["q"] + c["k"]) + 4.0 * D * _pairs(c) + _projection_flops(c)
    if c["kind"] in ("wan", "hunyuan"):
        nbytes = 2 * s * h * D * 2.0 + 4 * (h * D) ** 2 * 2.0 + n * D * 8.0
    else:
        nbytes = 4 * h * s * D * 2.0 + (2 * h * n * 8.0 if c["kind"] == "operators" else 0.0)
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """bf16 rows: an independent attention kernel (mma.sync, other tile shapes and summation order) on the
    same clustering is 0.9e-3 to 1.4e-3 away in the 2-norm and one bf16 step (0.008) in the largest element.
    Labels and maps: near ties only."""
    return {"rel": 5e-3, "max": 0.04, "differ": 1e-4}
