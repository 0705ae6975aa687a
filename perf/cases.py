"""The calls a denoiser makes into this package, as timed cases.

Every kind below is one attention sub-layer (or the part of it that this package
covers) of one of the denoisers: the state holds the weights, gains, tables,
caches, workspaces and output buffers that such a program keeps between calls,
and ``run`` makes the calls of one layer and one step.

    unet      SD1.5 transformer block at one U-Net level: self-attention with its
              projections, residual, cross-attention to the prompt (K/V projected
              once per prompt, or again in the call), residual, GEGLU feed-forward
              with its second linear layer, residual
    flux      Flux double-stream block: fused Q/K/V projection + RMSNorm + RoPE of
              the text and of the image stream, joint attention, both output
              projections
    single    Flux single-stream block whose Q, K, V are already projected: RMSNorm
              + RoPE pass, attention into the first columns of the wide row that
              the block's last linear layer reads
    joint     long-sequence joint attention (2048 px), text and image rows as two
              segments, two CFG branches in one call, or one rank's share of the heads
    extract   Qwen-Image first step over the text prefix: RoPE tables, projections,
              causal attention, output projection, K and V blended into the prefix cache
    cached    Qwen-Image later steps: image rows attend to the cached prefix and to
              themselves, with or without the prefix scale vectors
    gqa       grouped-query attention with a padded caption (Krea 2)
    sana      Sana ReLU linear attention, alone or after its three channel-major
              projections
    traced    joint attention with a text-steering bias and the head-averaged map of
              the image rows over the text keys

Activations are N(0, 1), weights N(0, 0.02), gains 1 + N(0, 0.02), as everywhere in
this repository's tests and benchmark.
"""
from __future__ import annotations

import math

import torch

import brodiffusion_b200 as bd

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # Bottom of the SD1.5 U-Net at 512 px (8 x 8 latent, head_dim 160): a few rows
        # against 1280-wide weights, seven dependent launches: latency.
        {"name": "unet_8x8", "kind": "unet", "tokens": 64, "channels": 1280, "heads": 8, "context": 77,
         "cached": True, "dtype": "fp16"},
        # A middle level (32 x 32, head_dim 80) whose prompt is projected in the call.
        {"name": "unet_32x32", "kind": "unet", "tokens": 1024, "channels": 640, "heads": 8, "context": 77,
         "cached": False, "dtype": "fp16"},
        # The top level (64 x 64, head_dim 40): most of a SD1.5 step's attention time.
        {"name": "unet_64x64", "kind": "unet", "tokens": 4096, "channels": 320, "heads": 8, "context": 77,
         "cached": True, "dtype": "fp16"},
        # First Qwen-Image step over a 256-token prompt: small, causal, many launches.
        {"name": "qwen_extract_256", "kind": "extract", "tokens": 256, "heads": 24, "dtype": "bf16"},
        # The other 39 steps at 1024 px.
        {"name": "qwen_cached_1024", "kind": "cached", "prefix": 256, "tokens": 4096, "heads": 24,
         "scaled": False, "dtype": "bf16"},
        # Flux.1 double-stream block at 1024 px.
        {"name": "flux_double_1024", "kind": "flux", "text": 512, "tokens": 4096, "heads": 24, "dtype": "bf16"},
        # Flux.1 single-stream block at a portrait size whose token count is no multiple of a tile.
        {"name": "flux_single_portrait", "kind": "single", "text": 333, "tokens": 2166, "heads": 24,
         "dtype": "bf16"},
        # Flux.1 at 2048 px, both CFG branches: the longest sequence this package is used on.
        {"name": "flux_joint_2048", "kind": "joint", "text": 512, "tokens": 16384, "batch": 2, "heads": 24,
         "dtype": "bf16"},
        # Krea-style grouped heads, captions padded to a fixed length, ragged image.
        {"name": "gqa_padded_caption", "kind": "gqa", "text": 512, "valid": 187, "tokens": 1530, "heads": 24,
         "kv_heads": 8, "dtype": "bf16"},
        # Sana 1.6B self-attention at 1024 px with its projections, one CFG branch.
        {"name": "sana_1024_projected", "kind": "sana", "tokens": 1024, "heads": 70, "batch": 1,
         "projected": True, "dtype": "bf16"},
        # The Sana core alone at 2048 px, both branches: bound by memory.
        {"name": "sana_core_4096", "kind": "sana", "tokens": 4096, "heads": 70, "batch": 2,
         "projected": False, "dtype": "bf16"},
        # Prompt-steering view of a Flux block at 512 px: bias in, map out.
        {"name": "flux_traced_512", "kind": "traced", "text": 256, "tokens": 1024, "heads": 24, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["unet", "unet", "flux", "single", "joint", "extract", "cached", "gqa", "sana", "traced"])
    if kind == "unet":
        channels = rng.choice([320, 640, 1280])
        most = {320: 9216, 640: 2304, 1280: 576}[channels]           # 768 px latents
        return {"kind": kind, "tokens": _log_int(rng, 48, most), "channels": channels, "heads": 8,
                "context": rng.choice([77, 154, rng.randint(20, 231)]), "cached": rng.random() < 0.6,
                "dtype": rng.choice(["fp16", "fp16", "bf16"])}
    heads = 24
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "flux":
        return {"kind": kind, "text": rng.choice([256, 512, rng.randint(40, 512)]),
                "tokens": _log_int(rng, 256, 6400), "heads": heads, "dtype": dtype}
    if kind == "single":
        return {"kind": kind, "text": rng.choice([256, 512, rng.randint(40, 512)]),
                "tokens": _log_int(rng, 200, 9000), "heads": heads, "dtype": dtype}
    if kind == "joint":
        return {"kind": kind, "text": rng.choice([256, 512]), "tokens": _log_int(rng, 1024, 16000),
                "batch": rng.choice([1, 2]), "heads": rng.choice([3, 6, 12, 24]), "dtype": dtype}
    if kind == "extract":
        return {"kind": kind, "tokens": _log_int(rng, 16, 1200), "heads": heads, "dtype": dtype}
    if kind == "cached":
        return {"kind": kind, "prefix": _log_int(rng, 24, 1500), "tokens": _log_int(rng, 256, 6400),
                "heads": heads, "scaled": rng.random() < 0.4, "dtype": dtype}
    if kind == "gqa":
        kv = rng.choice([2, 4, 8, 12])
        return {"kind": kind, "text": 512, "valid": rng.randint(8, 500), "tokens": _log_int(rng, 256, 8000),
                "heads": heads, "kv_heads": kv, "dtype": dtype}
    if kind == "sana":
        return {"kind": kind, "tokens": 8 * _log_int(rng, 32, 1024), "heads": rng.choice([36, 70]),
                "batch": rng.choice([1, 2]), "projected": rng.random() < 0.4, "dtype": "bf16"}
    return {"kind": "traced", "text": rng.choice([77, 256, 512]), "tokens": _log_int(rng, 256, 4096),
            "heads": heads, "dtype": dtype}


class _Make:
    """Seeded inputs on the GPU."""

    def __init__(self, case, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype = _DTYPES[case["dtype"]]

    def act(self, *shape):
        return torch.randn(*shape, device="cuda", dtype=self.dtype, generator=self.gen)

    def weight(self, *shape):
        return self.act(*shape) * 0.02

    def gain(self, n):
        return 1.0 + self.weight(n)

    def empty(self, *shape):
        return torch.empty(*shape, device="cuda", dtype=self.dtype)


def _flux_tables(text, tokens, hd):
    """cos/sin of ``text`` identity rows and a grid of at least ``tokens`` image rows."""
    w = max(1, int(math.sqrt(tokens)))
    h = -(-tokens // w)
    return bd.rope_tables_flux(text, h, w, hd)


# ----------------------------------------------------------------- unet
def _prepare_unet(c, m):
    n, ch, ctx = c["tokens"], c["channels"], c["context"]
    s = {"case": c, "x": m.act(n, ch)}
    for name in ("wq", "wk", "wv", "wo", "wq2", "wo2"):
        s[name] = m.weight(ch, ch)
    s["wk2"], s["wv2"], s["ctx"] = m.weight(ch, 768), m.weight(ch, 768), m.act(ctx, 768)
    s["bo"], s["bo2"], s["b_ff2"] = m.weight(ch), m.weight(ch), m.weight(ch)
    s["w_ff"], s["b_ff"], s["w_ff2"] = m.weight(8 * ch, ch), m.weight(8 * ch), m.weight(ch, 4 * ch)
    s["h1"], s["h2"], s["out"], s["ff"] = m.empty(n, ch), m.empty(n, ch), m.empty(n, ch), m.empty(n, 4 * ch)
    hd = ch // c["heads"]
    need = max(bd.qkvo_workspace_bytes(n, n, c["heads"], hd), bd.qkvo_workspace_bytes(n, ctx, c["heads"], hd))
    s["ws"] = torch.empty(need, device="cuda", dtype=torch.uint8)
    if c["cached"]:
        s["k"], s["v"] = m.empty(ctx, ch), m.empty(ctx, ch)
        bd.project_kv(s["ctx"], s["wk2"], s["wv2"], s["k"], s["v"])
    return s


def _run_unet(s):
    c = s["case"]
    nh = c["heads"]
    bd.qkvo_fwd(s["x"], None, s["wq"], s["wk"], s["wv"], s["wo"], s["bo"], nh, s["h1"], s["ws"])
    bd.add_inplace(s["h1"], s["x"])
    if c["cached"]:
        bd.qkvo_fwd(s["h1"], None, s["wq2"], None, None, s["wo2"], s["bo2"], nh, s["h2"], s["ws"],
                    k_cached=s["k"], v_cached=s["v"])
    else:
        bd.qkvo_fwd(s["h1"], s["ctx"], s["wq2"], s["wk2"], s["wv2"], s["wo2"], s["bo2"], nh, s["h2"], s["ws"])
    bd.add_inplace(s["h2"], s["h1"])
    bd.linear_geglu_fwd(s["h2"], s["w_ff"], s["b_ff"], s["ff"])
    bd.linear_fwd(s["ff"], s["w_ff2"], s["b_ff2"], s["out"])
    bd.add_inplace(s["out"], s["h2"])
    return s["h1"], s["h2"], s["out"]


def _work_unet(c):
    n, ch, ctx = c["tokens"], c["channels"], c["context"]
    flops = 2.0 * n * ch * ch * (4 + 2 + 8 + 4) + 4.0 * n * ch * (n + ctx)
    weights = (6 + 8 + 4) * ch * ch
    kv = 2 * ctx * ch
    if not c["cached"]:
        flops += 4.0 * ctx * 768 * ch
        kv = ctx * 768 + 2 * 768 * ch
    return {"bytes": 2.0 * (weights + kv + 4 * n * ch), "flops": flops}


# ----------------------------------------------------------------- flux
def _prepare_flux(c, m):
    hd, nh = 128, c["heads"]
    d = nh * hd
    s = {"case": c}
    s["cos"], s["sin"] = _flux_tables(c["text"], c["tokens"], hd)
    for t, rows in (("t", c["text"]), ("i", c["tokens"])):
        s["x" + t] = m.act(rows, d)
        for w in ("wq", "wk", "wv", "wo"):
            s[w + t] = m.weight(d, d)
        for b in ("bq", "bk", "bv", "bo"):
            s[b + t] = m.weight(d)
        s["gq" + t], s["gk" + t] = m.gain(hd), m.gain(hd)
        for o in ("q", "k", "v", "o", "y"):
            s[o + t] = m.empty(rows, d)
    return s


def _run_flux(s):
    c = s["case"]
    nh = c["heads"]
    for t, row0 in (("t", 0), ("i", c["text"])):
        bd.qkv_norm_rope_fwd(s["x" + t], s["wq" + t], s["wk" + t], s["wv" + t], s["q" + t], s["k" + t],
                             s["v" + t], nh, 128, gain_q=s["gq" + t], gain_k=s["gk" + t], cos=s["cos"],
                             sin=s["sin"], rope_row0=row0, bq=s["bq" + t], bk=s["bk" + t], bv=s["bv" + t])
    bd.sdpa_fwd([s["qt"], s["qi"]], [s["kt"], s["ki"]], [s["vt"], s["vi"]], [s["ot"], s["oi"]], nh)
    for t in ("t", "i"):
        bd.linear_fwd(s["o" + t], s["wo" + t], s["bo" + t], s["y" + t])
    return s["yt"], s["yi"]


def _work_flux(c):
    d, n = c["heads"] * 128, c["text"] + c["tokens"]
    return {"bytes": 2.0 * (8 * d * d + 2 * n * d) + 8.0 * n * 64, "flops": 8.0 * n * d * d + 4.0 * n * n * d}


# --------------------------------------------------------------- single
def _prepare_single(c, m):
    hd, nh = 128, c["heads"]
    d, n = nh * hd, c["text"] + c["tokens"]
    s = {"case": c, "gq": m.gain(hd), "gk": m.gain(hd)}
    s["cos"], s["sin"] = _flux_tables(c["text"], c["tokens"], hd)
    s["q"], s["k"], s["v"] = m.act(n, d), m.act(n, d), m.act(n, d)
    s["qr"], s["kr"], s["cat"] = m.empty(n, d), m.empty(n, d), m.empty(n, 5 * d)
    return s


def _run_single(s):
    c = s["case"]
    nh = c["heads"]
    bd.rmsnorm_rope([dict(x=s["q"], out=s["qr"], gain=s["gq"], cos=s["cos"], sin=s["sin"]),
                     dict(x=s["k"], out=s["kr"], gain=s["gk"], cos=s["cos"], sin=s["sin"])], nh, 128)
    out = s["cat"][:, :nh * 128]
    bd.sdpa_fwd(s["qr"], s["kr"], s["v"], out, nh)
    return out


def _work_single(c):
    d, n = c["heads"] * 128, c["text"] + c["tokens"]
    return {"bytes": 2.0 * 4 * n * d + 8.0 * n * 64, "flops": 4.0 * n * n * d}


# ---------------------------------------------------------------- joint
def _prepare_joint(c, m):
    hd, nh, b = 128, c["heads"], c["batch"]
    d, n = nh * hd, c["text"] + c["tokens"]
    s = {"case": c, "gains": [m.gain(hd) for _ in range(4)]}
    s["cos"], s["sin"] = _flux_tables(c["text"], c["tokens"], hd)
    s["q"], s["k"], s["v"] = m.act(b, n, d), m.act(b, n, d), m.act(b, n, d)
    s["qr"], s["kr"], s["out"] = m.empty(b, n, d), m.empty(b, n, d), m.empty(b, n, d)
    return s


def _run_joint(s):
    c = s["case"]
    nh, t = c["heads"], c["text"]
    for b in range(c["batch"]):
        jobs = []
        for x, r, gt, gi in (("q", "qr", 2, 0), ("k", "kr", 3, 1)):
            jobs.append(dict(x=s[x][b, :t], out=s[r][b, :t], gain=s["gains"][gt], cos=s["cos"], sin=s["sin"]))
            jobs.append(dict(x=s[x][b, t:], out=s[r][b, t:], gain=s["gains"][gi], cos=s["cos"], sin=s["sin"],
                             rope_row0=t))
        bd.rmsnorm_rope(jobs, nh, 128)
    seg = lambda x: [x[:, :t], x[:, t:]]  # noqa: E731
    bd.sdpa_fwd(seg(s["qr"]), seg(s["kr"]), seg(s["v"]), seg(s["out"]), nh)
    return s["out"]


def _work_joint(c):
    d, n = c["heads"] * 128, c["text"] + c["tokens"]
    return {"bytes": c["batch"] * 8.0 * n * d + 8.0 * n * 64, "flops": c["batch"] * 4.0 * n * n * d}


# ----------------------------------------------------- Qwen-Image steps
def _prepare_qwen(c, m):
    hd, nh = 128, c["heads"]
    d, n = nh * hd, c["tokens"]
    s = {"case": c, "x": m.act(n, d), "gq": m.gain(hd), "gk": m.gain(hd)}
    for w in ("wq", "wk", "wv", "wo"):
        s[w] = m.weight(d, d)
    for b in ("bq", "bk", "bv", "bo"):
        s[b] = m.weight(d)
    for o in ("q", "k", "v", "o", "y"):
        s[o] = m.empty(n, d)
    p = c["tokens"] if c["kind"] == "extract" else c["prefix"]
    s["pk"], s["pv"] = m.act(p, d), m.act(p, d)
    if c["kind"] == "cached":
        w = max(1, int(math.sqrt(n)))
        s["cos"], s["sin"] = bd.rope_tables_qwen([("text", p)], -(-n // w), w, hd)
        s["scale"] = {}
        if c["scaled"]:
            ks, vs = torch.ones(p + n, device="cuda"), torch.ones(p + n, device="cuda")
            ks[:p], vs[:p] = 0.5, 0.25
            s["scale"] = dict(key_scale=ks, val_scale=vs)
    return s


def _qwen_projections(s, cos, sin, row0):
    bd.qkv_norm_rope_fwd(s["x"], s["wq"], s["wk"], s["wv"], s["q"], s["k"], s["v"], s["case"]["heads"], 128,
                         gain_q=s["gq"], gain_k=s["gk"], cos=cos, sin=sin, rope_row0=row0, bq=s["bq"],
                         bk=s["bk"], bv=s["bv"])


def _run_extract(s):
    c = s["case"]
    # the tables are rebuilt at the start of every forward; the smallest target grid stands in here
    cos, sin = bd.rope_tables_qwen([("text", c["tokens"])], 8, 8, 128)
    _qwen_projections(s, cos, sin, 0)
    bd.sdpa_fwd(s["q"], s["k"], s["v"], s["o"], c["heads"], mask_mode=bd.MASK_CAUSAL)
    bd.linear_fwd(s["o"], s["wo"], s["bo"], s["y"])
    # blend_from: the stored prefix moves a quarter of the way towards this prompt's
    bd.axpby_inplace(s["pk"], s["k"], 0.75, 0.25)
    bd.axpby_inplace(s["pv"], s["v"], 0.75, 0.25)
    return s["y"], s["pk"], s["pv"]


def _run_cached(s):
    c = s["case"]
    _qwen_projections(s, s["cos"], s["sin"], c["prefix"])
    bd.sdpa_fwd(s["q"], [s["pk"], s["k"]], [s["pv"], s["v"]], s["o"], c["heads"], **s["scale"])
    bd.linear_fwd(s["o"], s["wo"], s["bo"], s["y"])
    return s["y"]


def _work_extract(c):
    d, n = c["heads"] * 128, c["tokens"]
    return {"bytes": 2.0 * (4 * d * d + 6 * n * d), "flops": 8.0 * n * d * d + 2.0 * n * (n + 1) * d}


def _work_cached(c):
    d, n, p = c["heads"] * 128, c["tokens"], c["prefix"]
    return {"bytes": 2.0 * (4 * d * d + 2 * n * d + 2 * p * d) + 8.0 * n * 64,
            "flops": 8.0 * n * d * d + 4.0 * n * (n + p) * d}


# ------------------------------------------------------------------ gqa
def _prepare_gqa(c, m):
    d, n = c["heads"] * 128, c["text"] + c["tokens"]
    dkv = c["kv_heads"] * 128
    mask = torch.ones(n, device="cuda")
    mask[c["valid"]:c["text"]] = 0.0
    return {"case": c, "q": m.act(n, d), "k": m.act(n, dkv), "v": m.act(n, dkv), "mask": mask, "o": m.empty(n, d)}


def _run_gqa(s):
    c = s["case"]
    bd.sdpa_fwd(s["q"], s["k"], s["v"], s["o"], c["heads"], num_kv_heads=c["kv_heads"], key_mask=s["mask"])
    return s["o"]


def _work_gqa(c):
    d, dkv, n = c["heads"] * 128, c["kv_heads"] * 128, c["text"] + c["tokens"]
    keys = n - (c["text"] - c["valid"])
    return {"bytes": 2.0 * (2 * n * d + 2 * keys * dkv) + 4.0 * n, "flops": 4.0 * n * keys * d}


# ----------------------------------------------------------------- sana
def _prepare_sana(c, m):
    d, n, b = c["heads"] * 32, c["tokens"], c["batch"]
    s = {"case": c, "o": m.empty(b, d, n)}
    if c["projected"]:
        s["x"] = m.act(b, n, d)
        s["w"] = [m.weight(d, d) for _ in range(3)]
        s["q"], s["k"], s["v"] = m.empty(b, d, n), m.empty(b, d, n), m.empty(b, d, n)
    else:
        s["q"], s["k"], s["v"] = m.act(b, d, n), m.act(b, d, n), m.act(b, d, n)
    return s


def _run_sana(s):
    c = s["case"]
    if c["projected"]:
        for b in range(c["batch"]):
            for w, y in zip(s["w"], ("q", "k", "v")):
                bd.linear_fwd(w, s["x"][b], None, s[y][b])       # (D, D) . (N, D)^T -> channel-major (D, N)
    bd.linear_attn_relu_fwd(s["q"], s["k"], s["v"], s["o"], c["heads"], 32)
    return s["o"]


def _work_sana(c):
    d, n, b = c["heads"] * 32, c["tokens"], c["batch"]
    flops = 4.0 * b * n * d * 33
    if c["projected"]:
        return {"bytes": 2.0 * (2 * b * n * d + 3 * d * d), "flops": flops + 6.0 * b * n * d * d}
    return {"bytes": 8.0 * b * n * d, "flops": flops}


# --------------------------------------------------------------- traced
def _prepare_traced(c, m):
    d, t, n = c["heads"] * 128, c["text"], c["tokens"]
    s = {"case": c, "bias": torch.zeros(n, t, device="cuda")}
    s["bias"][:, t // 4:t // 2] = torch.randn(n, 1, device="cuda", generator=m.gen)   # a steered phrase
    for x in ("q", "k", "v"):
        s[x] = [m.act(t, d), m.act(n, d)]
    s["o"] = [m.empty(t, d), m.empty(n, d)]
    return s


def _run_traced(s):
    c = s["case"]
    amap = bd.sdpa_traced_fwd(s["q"], s["k"], s["v"], s["o"], c["heads"], bias=s["bias"], bias_row0=c["text"],
                              map_row0=c["text"], map_rows=c["tokens"], map_cols=c["text"])
    return s["o"][0], s["o"][1], amap


def _work_traced(c):
    d, t, n = c["heads"] * 128, c["text"], c["text"] + c["tokens"]
    return {"bytes": 8.0 * n * d + 8.0 * c["tokens"] * t, "flops": 4.0 * n * n * d}


_PREPARE = {"unet": _prepare_unet, "flux": _prepare_flux, "single": _prepare_single, "joint": _prepare_joint,
            "extract": _prepare_qwen, "cached": _prepare_qwen, "gqa": _prepare_gqa, "sana": _prepare_sana,
            "traced": _prepare_traced}
_RUN = {"unet": _run_unet, "flux": _run_flux, "single": _run_single, "joint": _run_joint, "extract": _run_extract,
        "cached": _run_cached, "gqa": _run_gqa, "sana": _run_sana, "traced": _run_traced}
_WORK = {"unet": _work_unet, "flux": _work_flux, "single": _work_single, "joint": _work_joint,
         "extract": _work_extract, "cached": _work_cached, "gqa": _work_gqa, "sana": _work_sana,
         "traced": _work_traced}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, _Make(case, seed))


def run(state):
    return _RUN[state["case"]["kind"]](state)


def work(case):
    return _WORK[case["kind"]](case)


def tolerance(case):
    """Four times what the outputs of all kinds differ by from the same chain in 64-bit
    arithmetic: rel 3.6e-3, max 3.6e-2 with BF16 storage, rel 4.8e-4, max 2.4e-3 with
    FP16 (intermediates and outputs are rounded to the storage type)."""
    return {"rel": 1.4e-2, "max": 0.15} if case["dtype"] == "bf16" else {"rel": 2e-3, "max": 1e-2}
