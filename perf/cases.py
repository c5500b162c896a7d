"""Performance cases of the token-sparse attention path: the calls a video-DiT sampler makes through the public API.

A denoising run consists of a few dense steps, anchor steps (dense pass with LSE, Fast PDDP grouping, group mass, token
selection, residual), occasional selection updates, and mostly reuse steps (one gather-KV attention call per layer).
Every case is one such call.  Sizes: the 21 x 39 x 40 latent grid with 24 heads and 2,048 selected tokens, the
21 x 72 x 65 grid with 40 heads and 4,096, the 4,096-token two-head case and the head dimensions 64 / 128 / 144 that the
benchmark and the tests use, plus short and ragged sequences.

Inputs are clustered latents: token t carries the centroid of its run of neighbouring tokens, scaled per head so that
some heads attend sharply and others broadly, plus noise; V is Gaussian.  Everything comes from the seed alone.
"""

import math

import torch

from mcsparse_b200.h3.ulysses_layer import UlyssesDiTAttentionLayer
from mcsparse_b200.kernels.flash_mcsa.ops.flash_sparse_attn.cute import flash_attn_gather_kv_func
from mcsparse_b200.kernels.flash_mcsa.ops.flash_sparse_attn.cute.interface import flash_attn_gather_kv_fp8_func
from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention
from mcsparse_b200.kernels.flash_mcsa.pca_group import pca_group_perm
from mcsparse_b200.kernels.flash_mcsa.token_sparse import (TokenSparseConfig, TokenSparseContext, select_topk_with_sinks)

SINKS = 4                      # forced tokens at the start of the sequence
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # the smallest reuse call: 128 groups of 64 queries, 512 tokens each; launch and host latency
        {"name": "attn_small_d64", "kind": "attn", "H": 2, "L": 4096, "D": 64, "K": 512, "rows": 64, "dtype": "bf16",
         "perm": False, "residual": True},
        # the reuse call of the single-GPU video DiT: most layers of most steps are this call
        {"name": "attn_dit", "kind": "attn", "H": 24, "L": 32760, "D": 128, "K": 2048, "rows": 128, "dtype": "bf16",
         "perm": True, "residual": True},
        # a reuse call at the other head dimension of the reference's dispatch, fp16, odd length
        {"name": "attn_d144", "kind": "attn", "H": 8, "L": 20475, "D": 144, "K": 3072, "rows": 128, "dtype": "fp16",
         "perm": True, "residual": True},
        # the long video in FP8: the eight heads that one of five GPUs holds
        {"name": "attn_long_fp8", "kind": "attn_fp8", "H": 8, "L": 98280, "D": 128, "K": 4096, "residual": True},
        # a dense step (or dense layer) of the single-GPU video DiT
        {"name": "dense_dit", "kind": "dense", "H": 24, "L": 32760, "D": 128, "dtype": "bf16"},
        # anchor step of the same model: everything that the following reuse steps live on
        {"name": "anchor_dit", "kind": "anchor", "H": 24, "L": 32760, "D": 128, "topk": 0.0625, "dtype": "bf16"},
        # anchor step of a short clip with a ragged length and smaller heads
        {"name": "anchor_short_d64", "kind": "anchor", "H": 12, "L": 4700, "D": 64, "topk": 0.25, "dtype": "fp16"},
        # selection update with budgets by mass (top-p with a top-k floor) and per-group lengths
        {"name": "update_topp", "kind": "update", "H": 8, "L": 16380, "D": 128, "topk": 0.1, "topp": 0.7, "dtype": "bf16"},
        # one denoising step of four layers of a short clip in reuse mode: kernels and the host between them
        {"name": "reuse_step_short", "kind": "reuse", "H": 24, "L": 4680, "D": 128, "topk": 0.25, "layers": 4,
         "dtype": "bf16"},
        # token selection of the long video from given masses (rows longer than 32,768)
        {"name": "select_long", "kind": "select", "H": 5, "M": 768, "L": 98280, "K": 4096},
        # query grouping of the single-GPU video DiT
        {"name": "group_dit", "kind": "group", "H": 24, "L": 32760, "D": 128, "dtype": "bf16"},
        # the whole attention layer of the long video on one GPU, projections included
        {"name": "layer_long", "kind": "layer", "heads": 40, "D": 128, "F": 21, "Y": 72, "X": 65, "K": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tiles(n, L):
    """A token budget: a whole number of 128-token tiles that fits the sequence."""
    return max(128, min(n // 128 * 128, L // 128 * 128))


def draw(rng):
    kind = rng.choice(["attn", "attn", "attn", "attn_fp8", "dense", "anchor", "update", "reuse", "select", "group", "layer"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "attn":
        L = _log(rng, 4000, 98280)
        H = _log(rng, 1, max(1.0, min(40.0, 800000 / L)))
        rows = 128 if L > 16384 else rng.choice([64, 128, 128])
        return {"kind": kind, "H": H, "L": L, "D": rng.choice([64, 96, 128, 128, 128, 144, 192]), "K": _tiles(_log(rng, 256, 4096), L),
                "rows": rows, "dtype": dtype, "perm": rng.random() < 0.7, "residual": rng.random() < 0.7}
    if kind == "attn_fp8":
        L = _log(rng, 8000, 98280)
        return {"kind": kind, "H": _log(rng, 2, min(40.0, 800000 / L)), "L": L, "D": rng.choice([128, 128, 160]),
                "K": _tiles(_log(rng, 512, 4096), L), "residual": rng.random() < 0.7}
    if kind == "dense":
        L = _log(rng, 600, 32760)
        return {"kind": kind, "H": _log(rng, 2, 24), "L": L, "D": rng.choice([64, 128, 128]), "dtype": dtype}
    if kind in ("anchor", "update"):
        L = _log(rng, 4100, 32760)
        c = {"kind": kind, "H": _log(rng, 2, 24), "L": L, "D": rng.choice([64, 128, 128]), "topk": round(rng.uniform(0.06, 0.25), 3),
             "dtype": dtype}
        if kind == "update":
            c["topp"] = round(rng.uniform(0.5, 0.8), 2)
        return c
    if kind == "reuse":
        L = _log(rng, 4100, 16380)
        return {"kind": kind, "H": _log(rng, 4, 24), "L": L, "D": rng.choice([64, 128, 128]), "topk": round(rng.uniform(0.1, 0.25), 3),
                "layers": rng.randint(2, 6), "dtype": dtype}
    if kind == "select":
        L = _log(rng, 4096, 98280)
        return {"kind": kind, "H": _log(rng, 1, 24), "M": min(768, math.ceil(L / 128)), "L": L, "K": _tiles(_log(rng, 256, 8192), L)}
    if kind == "group":
        L = _log(rng, 1000, 98280)
        return {"kind": kind, "H": _log(rng, 1, min(24.0, 790000 / L)), "L": L, "D": rng.choice([64, 128, 128]), "dtype": dtype}
    return {"kind": kind, "heads": rng.choice([4, 8, 16, 24]), "D": 128, "F": rng.randint(5, 21), "Y": rng.randint(20, 72),
            "X": rng.randint(20, 65), "K": rng.choice([1024, 2048])}


# ------------------------------------------------------------------------------------------------- inputs
def _latents(case, seed, L=None):
    """q, k, v (1, L, H, D) on the GPU.  Runs of about L / 200 neighbouring tokens share one of 64 centroids; the sharpness
    of a head's attention differs from head to head."""
    H, D, L = case["H"], case["D"], L or case["L"]
    dt = DTYPES.get(case.get("dtype", "bf16"))
    g = torch.Generator(device="cuda").manual_seed(seed * 1009 + 7)
    run = max(8, L // 200)
    cid = ((torch.arange(L, device="cuda") // run) * 37) % 64
    amp = torch.linspace(0.55, 0.85, H, device="cuda").view(H, 1, 1) * (128.0 / D) ** 0.25
    cent = amp * torch.randn(H, 64, D, generator=g, device="cuda")
    q = torch.empty(1, L, H, D, dtype=dt, device="cuda")
    k, v = torch.empty_like(q), torch.empty_like(q)
    for h in range(H):
        c = cent[h][cid]
        q[0, :, h] = c + 0.3 * torch.randn(L, D, generator=g, device="cuda")
        k[0, :, h] = c + 0.3 * torch.randn(L, D, generator=g, device="cuda")
        v[0, :, h] = torch.randn(L, D, generator=g, device="cuda")
    return q, k, v, cid, g


def _grouping(case, cid, g):
    """A permutation per head that brings tokens of one centroid together, as the query grouping does: (H, L) int64."""
    L = case["L"]
    return torch.stack([torch.argsort(cid + 0.9 * torch.rand(L, generator=g, device="cuda")) for _ in range(case["H"])])


def _indices(q, k, perm, rows, K):
    """Per head and query group: the sink tokens and the keys that score best against the group's mean query, ascending."""
    H, L = q.shape[2], q.shape[1]
    M = math.ceil(L / rows)
    out = torch.empty(1, H, M, K, dtype=torch.int32, device="cuda")
    for h in range(H):
        x = q[0, :, h] if perm is None else q[0, perm[h], h]
        pad = torch.zeros(M * rows, x.shape[1], device="cuda")
        pad[:L] = x
        s = pad.view(M, rows, -1).mean(1) @ k[0, :, h].float().t()
        s[:, :SINKS] = float("inf")
        out[0, h] = s.topk(K, dim=-1).indices.sort(dim=-1).values
    return out


def _spread_indices(H, M, L, K, g):
    """Ascending index lists spread over the whole sequence, one random token from each of K equal strata."""
    lo = torch.arange(K, device="cuda") * L // K
    width = (torch.arange(1, K + 1, device="cuda") * L // K - lo).float()
    out = torch.empty(1, H, M, K, dtype=torch.int32, device="cuda")
    for h in range(H):
        out[0, h] = (lo + (torch.rand(M, K, generator=g, device="cuda") * width).long()).to(torch.int32)
    return out


def _config(case):
    c = dict(topk=case["topk"], pca_reorder=True, sink_ranges=[(0, SINKS)])
    if case["kind"] == "anchor":
        return TokenSparseConfig(calibrate_steps=[0], full_steps=[0], bias_correction=True, **c)
    if case["kind"] == "update":
        return TokenSparseConfig(calibrate_steps=[0], update_steps=[1], selection_mode="topk_topp", topp=case["topp"], **c)
    return TokenSparseConfig(calibrate_steps=[0], full_steps=[0], bias_correction=True, **c)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "select":
        g = torch.Generator(device="cuda").manual_seed(seed * 1009 + 7)
        H, M, L = case["H"], case["M"], case["L"]
        # attention masses fall off roughly log-normally; a tenth of the keys underflow to nothing
        s = torch.empty(1, H, M, L, device="cuda")
        for h in range(H):
            x = torch.randn(M, L, generator=g, device="cuda")
            s[0, h] = torch.where(x < -1.28, 0.0, torch.exp(2.0 * x) / L)
        return {"case": case, "scores": s}
    if kind == "layer":
        g = torch.Generator(device="cuda").manual_seed(seed * 1009 + 7)
        H, D, K = case["heads"], case["D"], case["K"]
        grid = (case["F"], case["Y"], case["X"])
        L, hidden = grid[0] * grid[1] * grid[2], H * D
        w = {n: (torch.randn(hidden, hidden, generator=g, device="cuda") / math.sqrt(hidden)).to(torch.bfloat16)
             for n in ("wq", "wk", "wv", "wo")}
        for n in ("gq", "gk"):
            w[n] = 1.0 + 0.1 * torch.randn(D, generator=g, device="cuda")
        layer = UlyssesDiTAttentionLayer(None, hidden, H, D, grid, w, torch.device("cuda"), heads_per_chunk=8 if H % 8 == 0 else 4)
        M = math.ceil(L / 128)
        res = torch.empty(1, H, L, D, dtype=torch.bfloat16, device="cuda")
        for h in range(H):
            res[0, h] = 0.1 * torch.randn(L, D, generator=g, device="cuda")
        layer.set_metadata(_spread_indices(H, M, L, _tiles(K, L), g), res)
        x = torch.randn(L, hidden, generator=g, device="cuda", dtype=torch.bfloat16)
        return {"case": case, "layer": layer, "x": x}
    if kind == "reuse":
        layers = []
        ctx = TokenSparseContext(_config(case), num_layers=case["layers"])
        for li in range(case["layers"]):
            q, k, v = (t.transpose(1, 2) for t in _latents(case, seed * 31 + li)[:3])
            ctx.forward(li, q, k, v)                     # the anchor step that the reuse steps live on
            layers.append((q, k, v))
        ctx.step()
        return {"case": case, "ctx": ctx, "layers": layers}
    q, k, v, cid, g = _latents(case, seed)
    if kind == "group":
        return {"case": case, "x": q[0].transpose(0, 1)}
    if kind in ("dense", "anchor", "update"):
        st = {"case": case, "qkv": tuple(t.transpose(1, 2) for t in (q, k, v))}
        if kind != "dense":
            st["ctx"] = TokenSparseContext(_config(case), num_layers=1)
        if kind == "update":
            st["ctx"].forward(0, *st["qkv"])             # the anchor step whose LSE and grouping the update reuses
            st["ctx"].step()
        return st
    perm = _grouping(case, cid, g) if case.get("perm") else None
    gi = _indices(q, k, perm, case.get("rows", 128), case["K"])
    res = None
    if case["residual"]:
        dt = torch.bfloat16 if kind == "attn_fp8" else q.dtype
        res = torch.empty(1, case["H"], case["L"], case["D"], dtype=dt, device="cuda")
        for h in range(case["H"]):
            res[0, h] = 0.1 * torch.randn(case["L"], case["D"], generator=g, device="cuda")
    if kind == "attn":
        return {"case": case, "qkv": (q, k, v), "gi": gi, "res": res, "perm": perm}
    x8, sc = [], []
    for t in (q, k, v):                                  # per-head symmetric quantisation
        s = t.float().abs().amax(dim=(1, 3)).clamp_min(1e-12) / 448.0
        x8.append((t.float() / s[:, None, :, None]).to(torch.float8_e4m3fn))
        sc.append(s)
    M = gi.shape[2]
    qk = (sc[0] * sc[1] * (math.log2(math.e) / math.sqrt(case["D"])))[:, :, None].expand(1, case["H"], M).contiguous()
    return {"case": case, "qkv": tuple(x8), "gi": gi, "res": res, "qk": qk, "sv": sc[2].contiguous()}


# --------------------------------------------------------------------------------------------------- passes
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "attn":
        out, lse = flash_attn_gather_kv_func(*state["qkv"], state["gi"], residual=state["res"], perm=state["perm"],
                                             group_rows=case["rows"], return_lse=True)
        return out, lse
    if kind == "attn_fp8":
        return flash_attn_gather_kv_fp8_func(*state["qkv"], state["gi"], state["qk"], state["sv"], residual=state["res"],
                                             return_lse=True)
    if kind == "dense":
        return full_attention(*state["qkv"])
    if kind == "group":
        return pca_group_perm(state["x"])
    if kind == "select":
        return select_topk_with_sinks(state["scores"], case["K"], [(0, SINKS)])
    if kind == "layer":
        return state["layer"].forward(state["x"])
    ctx = state["ctx"]
    if kind == "reuse":
        outs = [ctx.forward(li, *qkv) for li, qkv in enumerate(state["layers"])]
        ctx.step()
        return outs
    out = ctx.forward(0, *state["qkv"])
    c = ctx.caches[0]
    if kind == "update":
        return out, c._cached_lengths                    # (the index list's width follows the data; the output depends on all of it)
    return out, c._cached_residual, c._cached_lse, c._cached_perm, c._cached_indices


# ------------------------------------------------------------------------------------------ cost and tolerance
def work(case):
    kind = case["kind"]
    if kind == "select":
        rows = case["H"] * case["M"]
        return {"bytes": 4.0 * rows * (case["L"] + case["K"]), "flops": 0.0}
    if kind == "layer":
        hd, L = case["heads"] * case["D"], case["F"] * case["Y"] * case["X"]
        K = _tiles(case["K"], L)
        # x in, out, four weights, residual, indices; four projections and the attention on the selected tokens
        return {"bytes": 2.0 * (3 * L * hd + 4 * hd * hd) + 4.0 * case["heads"] * math.ceil(L / 128) * K,
                "flops": 8.0 * L * hd * hd + 4.0 * L * K * hd}
    H, L, D = case["H"], case["L"], case["D"]
    t = 2.0 * H * L * D                                  # one (L, H, D) tensor of 16-bit values
    if kind == "group":
        return {"bytes": t + 8.0 * H * L, "flops": 0.0}
    if kind == "dense":
        return {"bytes": 4 * t, "flops": 4.0 * L * L * D * H}
    if kind in ("attn", "attn_fp8"):
        io = (4 * t if kind == "attn" else 2.5 * t) + (t if case["residual"] else 0.0)
        meta = 4.0 * H * math.ceil(L / case.get("rows", 128)) * case["K"] + 4.0 * H * L + (8.0 * H * L if case.get("perm") else 0.0)
        return {"bytes": io + meta, "flops": 4.0 * L * case["K"] * D * H}
    K = min(L, math.ceil(case["topk"] * L / 128) * 128)
    meta = 4.0 * H * math.ceil(L / 128) * K
    sparse = 4.0 * L * K * D * H
    if kind == "reuse":
        return {"bytes": case["layers"] * (5 * t + meta + 8.0 * H * L), "flops": case["layers"] * sparse}
    if kind == "update":                                 # group mass, selection, sparse attention (at the top-k floor)
        return {"bytes": 4 * t + meta + 12.0 * H * L, "flops": 2.0 * L * L * D * H + sparse}
    return {"bytes": 5 * t + meta + 12.0 * H * L, "flops": 6.0 * L * L * D * H + sparse}


def tolerance(case):
    """About four times the distance to the same path in 64 bits, measured at the listed sizes (2-norm; largest)."""
    kind = case["kind"]
    if kind == "select":
        return "exact"                                   # a pure function of the fp32 scores
    if kind == "group":
        return {"rel": 0.0, "max": 0.0, "differ": 0.01}  # 2.7e-4 of the positions in bf16, 5.3e-3 in fp16 (near-ties)
    if kind == "attn_fp8":
        return {"rel": 0.03, "max": 0.9}                 # 7.2e-3; 0.28 (three mantissa bits per probability)
    if kind in ("anchor", "update"):
        # the residual is a difference of two close results: 8.6e-3; 0.15.  Selection: 3.5e-3 of the positions (near-ties)
        return {"rel": 0.03, "max": 0.6, "differ": 0.01}
    if case.get("dtype") == "fp16":
        return {"rel": 1.2e-3, "max": 0.01}              # 2.3e-4; 1.9e-3
    return {"rel": 0.01, "max": 0.12}                    # 2.3e-3; 2.9e-2
