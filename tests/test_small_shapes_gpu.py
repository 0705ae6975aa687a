"""Calls whose shape decides the route: head dims above 128 (mma.sync kernel), linear
layers whose K blocks are shared by a cluster or whose tiles are shared by a pair of CTAs,
and map blocks at the edges of their tiles and segments.  References: the CPU oracle."""
import numpy as np
import pytest
import torch

import gpu_util as G
import synth

pytestmark = pytest.mark.gpu


def _acts(shapes, seed, storage):
    return [synth.activations(s, seed + i, storage) for i, s in enumerate(shapes)]


# Rows and keys around the 16-row / 16-key tiles, one and two row tiles per CTA (the
# second where the call fills the SMs), both padded widths, every option of the kernel.
# The probabilities keep FP32 and only the output is rounded: half an ulp of a value
# below 4 is 2^-8 in BF16 and 2^-10 in FP16.
@pytest.mark.parametrize("storage", ["bf16", "fp16"])
@pytest.mark.parametrize("hd,nh,Lq,Lk,opt", [
    (160, 8, 64, 64, ""), (160, 8, 1, 1, ""), (160, 2, 17, 15, "mask"), (160, 3, 33, 129, "causal"),
    (160, 8, 576, 577, "mask"), (160, 8, 600, 77, "scale"), (136, 2, 70, 49, "scale"), (256, 2, 48, 130, "causal"),
    (168, 5, 31, 200, "mask"), (200, 1, 16, 16, "scale"), (160, 2, 40, 24, "causal")])
def test_head_dims_above_128(bd, oracle, storage, hd, nh, Lq, Lk, opt):
    q, k, v = _acts([(Lq, nh * hd), (Lk, nh * hd), (Lk, nh * hd)], 9500 + hd + Lq, storage)
    kw = {}
    if opt == "causal":
        kw["mask_mode"] = 1
    if opt == "mask":
        kw["key_mask"] = (synth.uniform01(Lk, 9501) > 0.3).astype(np.float32)
    if opt == "scale":
        kw["key_scale"] = 0.5 + synth.uniform01(Lk, 9502).astype(np.float32)
        kw["val_scale"] = (100.0 * synth.uniform01(Lk, 9503)).astype(np.float32) ** 2 if storage == "fp16" else \
            synth.uniform01(Lk, 9503).astype(np.float32)
        if storage == "fp16":
            v = synth.round_fp16(v * 1e-3)
    dt = torch.bfloat16 if storage == "bf16" else torch.float16
    got = G.sdpa(bd, q, k, v, nh, dtype=dt, **kw)
    ks, vs = kw.pop("key_scale", None), kw.pop("val_scale", None)
    if ks is not None:
        k, v = k * ks[:, None], v * vs[:, None]
    ref = oracle.sdpa(q, k, v, nh, **kw)
    half_ulp = np.exp2(np.ceil(np.log2(np.abs(ref).max() + 1e-9))) * (2.0 ** -9 if storage == "bf16" else 2.0 ** -12)
    assert np.abs(got - ref).max() <= half_ulp + 1e-4 * np.abs(ref).max()


def test_head_dims_above_128_probabilities_near_one(bd):
    """Two keys of almost the same score and opposite values: the output is V * tanh(d / 2), all of it what
    the second probability 1 - d lacks to one.  Root mean square error of that probability over 256 rows:
    2^-23 / sqrt(12) from its two parts, as much from the exponential and less from the output's
    rounding, 0.6e-7 in all; an exponent rounded at 2^-20 makes 1.9e-7."""
    hd, rows, big = 160, 256, 32768.0
    d = np.exp2(-14.0 + 2.0 * np.arange(rows) / rows)
    c = synth.round_fp16((d * np.sqrt(hd)).astype(np.float32))
    q = np.zeros((rows, hd), np.float32)
    q[:, 0] = c
    k = np.zeros((2, hd), np.float32)
    k[1, 0] = -1.0
    v = np.full((2, hd), big, np.float32)
    v[1] = -big
    got = G.sdpa(bd, q, k, v, 1, dtype=torch.float16)
    err = (got[:, 0].astype(np.float64) / big - np.tanh(c.astype(np.float64) / np.sqrt(hd) / 2.0)) * 2.0
    assert np.sqrt(np.mean(err ** 2)) < 1e-7


# Value scales far from one with FP16 values: a scale of 1e8 on a key nobody sees, scales of 1e-8 on values
# near 5e4, scales that span twelve decades.  Only the output is rounded (bound as above, for the largest
# value of a row's 160 columns: what cancels there leaves FP32 errors of that size).
@pytest.mark.parametrize("hd,nh,Lq,Lk", [(160, 2, 40, 50), (160, 8, 600, 36), (256, 2, 20, 4)])
@pytest.mark.parametrize("kind", ["masked", "small", "wide"])
def test_head_dims_above_128_value_scales_far_from_one(bd, oracle, hd, nh, Lq, Lk, kind):
    q, k, v = _acts([(Lq, nh * hd), (Lk, nh * hd), (Lk, nh * hd)], 9540 + hd, "fp16")
    scale = 0.5 + 0.5 * synth.uniform01(Lk, 9541).astype(np.float32)
    mask = np.ones(Lk, np.float32)
    if kind == "masked":
        scale[1], mask[1] = 1e8, 0.0
    elif kind == "small":
        v = synth.round_fp16((5e4 * (0.5 + 0.5 * synth.uniform01(v.size, 9542))).astype(np.float32).reshape(v.shape))
        scale *= 1e-8
    else:
        scale *= np.power(10.0, np.linspace(-10, 2, Lk)).astype(np.float32)
        v = synth.round_fp16(v * 16.0)
    got = G.sdpa(bd, q, k, v, nh, dtype=torch.float16, key_mask=mask, val_scale=scale)
    ref = oracle.sdpa(q, k, v * scale[:, None], nh, key_mask=mask)
    half_ulp = np.exp2(np.maximum(np.floor(np.log2(np.abs(ref) + 1e-30)), -14.0) - 11.0)
    top = np.abs(ref.reshape(Lq, nh, hd)).max(axis=2, keepdims=True)
    slack = np.broadcast_to(1e-4 * top, (Lq, nh, hd)).reshape(Lq, nh * hd)
    assert (np.abs(got - ref) <= half_ulp + slack).all()


def test_head_dims_above_128_segments_and_groups(bd, oracle):
    """Two segments on both sides whose border is inside a tile, two query heads per K/V head."""
    hd, nh, nkv = 160, 4, 2
    q = synth.activations((45, nh * hd), 9520)
    k, v = _acts([(39, nkv * hd)] * 2, 9521, "bf16")
    tq, tk, tv = G.dev(q), G.dev(k), G.dev(v)
    out = torch.full_like(tq, float("nan"))
    bd.sdpa_fwd([tq[:21], tq[21:]], [tk[:19], tk[19:]], [tv[:19], tv[19:]], [out[:21], out[21:]], nh, num_kv_heads=nkv)
    assert bd.device_status() == 0
    rep = lambda x: np.repeat(x.reshape(-1, nkv, hd), nh // nkv, axis=1).reshape(x.shape[0], -1)
    G.check(G.host(out), oracle.sdpa(q, rep(k), rep(v), nh), what="segments and groups, head_dim 160")


# Infinite and NaN values stay what a sum of products makes of them, in their own columns only; the
# key that carries them is in the first, a middle or the last (ragged) chunk of sixteen.
@pytest.mark.parametrize("storage", ["bf16", "fp16"])
@pytest.mark.parametrize("hd,Lq,Lk,key", [(160, 40, 70, 3), (160, 600, 70, 37), (136, 17, 70, 69), (256, 20, 33, 32)])
def test_head_dims_above_128_values_that_are_not_finite(bd, oracle, storage, hd, Lq, Lk, key):
    nh = 8 if Lq > 100 else 2
    q, k, v = _acts([(Lq, nh * hd), (Lk, nh * hd), (Lk, nh * hd)], 9530 + hd, storage)
    ref = oracle.sdpa(q, k, v, nh)
    other = (key + 29) % Lk
    for col, vals in ((1, (np.inf,)), (7, (-np.inf,)), (hd - 1, (np.inf, -np.inf)), (64, (np.nan,)), (hd + 5, (np.inf, np.inf))):
        for row, val in zip((key, other), vals):
            v[row, col] = val
        ref[:, col] = sum(vals) if len(set(vals)) == 1 else np.nan
    got = G.sdpa(bd, q, k, v, nh, dtype=torch.bfloat16 if storage == "bf16" else torch.float16)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(got[inf], ref[inf])
    fin = np.isfinite(ref)
    half_ulp = np.exp2(np.ceil(np.log2(np.abs(ref[fin]).max()))) * (2.0 ** -9 if storage == "bf16" else 2.0 ** -12)
    assert np.abs(got[fin] - ref[fin]).max() <= half_ulp + 1e-4 * np.abs(ref[fin]).max()


# Few output tiles, so that 2, 4 or 8 CTAs share a tile: ragged rows and columns, K not a
# multiple of a K block, the smallest K that is split (eleven blocks) and shorter ones that are not
# (tests/test_gemm_plan.py has the rule).
@pytest.mark.parametrize("M,N,K", [(64, 1280, 1280), (64, 1280, 5120), (1, 72, 2048), (77, 1280, 768), (130, 200, 1000),
                                   (256, 3072, 3072), (128, 64, 384), (128, 64, 320), (300, 640, 2560),
                                   (128, 64, 648), (128, 64, 640)])
def test_linear_split_over_a_cluster(bd, oracle, M, N, K):
    x, w, b = synth.activations((M, K), 9600 + M), synth.weights((N, K), 9601 + N), synth.weights((N,), 9602)
    for bias in (b, None):
        y = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        bd.linear_fwd(G.dev(x), G.dev(w), G.dev(bias) if bias is not None else None, y)
        assert bd.device_status() == 0
        ref = oracle.linear(x, w, bias)
        # half an ulp of the largest output, and FP32 sums in another order
        assert np.abs(G.host(y) - ref).max() <= np.abs(ref).max() * (2.0 ** -8 + 1e-5)


# Few rows: GEGLU is never split, these take 64 columns (the ragged ones) or pairs.
@pytest.mark.parametrize("B,Din,Dout", [(64, 1280, 5120), (33, 1280, 264), (130, 520, 72)])
def test_geglu_few_rows(bd, oracle, B, Din, Dout):
    x, w = synth.activations((B, Din), 9700, "fp16"), synth.weights((2 * Dout, Din), 9701, "fp16")
    b = synth.weights((2 * Dout,), 9702, "fp16")
    y = torch.full((B, Dout), float("nan"), device="cuda", dtype=torch.float16)
    bd.linear_geglu_fwd(G.dev(x, torch.float16), G.dev(w, torch.float16), G.dev(b, torch.float16), y)
    assert bd.device_status() == 0
    ref = oracle.linear_geglu(x, w, b)
    assert np.abs(G.host(y) - ref).max() <= 0.01 * np.abs(ref).max() + 0.008   # the reference's own bound


# Tiles of 256 x 256 shared by two CTAs: row counts that leave the second CTA empty or
# part-filled, more than one group of sixteen row blocks, K not a multiple of a K block.
@pytest.mark.parametrize("M,N,K", [(4500, 1280, 72), (9473, 512, 200), (2304, 2560, 136)])
def test_linear_on_cta_pairs(bd, oracle, M, N, K):
    x, w, b = synth.activations((M, K), 9650 + M), synth.weights((N, K), 9651 + N), synth.weights((N,), 9652)
    y = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    bd.linear_fwd(G.dev(x), G.dev(w), G.dev(b), y)
    assert bd.device_status() == 0
    ref = oracle.linear(x, w, b)
    assert np.abs(G.host(y) - ref).max() <= np.abs(ref).max() * (2.0 ** -8 + 1e-5)


@pytest.mark.parametrize("hd,nh,rows", [(128, 24, 16), (128, 4, 130), (64, 3, 77), (64, 8, 300), (128, 2, 1)])
def test_qkv_norm_rope_few_rows(bd, oracle, hd, nh, rows):
    D, d_in = nh * hd, 1024
    x = synth.activations((rows, d_in), 9800)
    ws = [synth.weights((D, d_in), 9801 + i) for i in range(3)]
    bs = [synth.weights((D,), 9810 + i) for i in range(3)]
    gq, gk = synth.gains(hd, 9820), synth.gains(hd, 9821)
    ang = synth.uniform01(rows * hd // 2, 9822).reshape(rows, hd // 2) * 6.0
    cos, sin = np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)
    outs = [torch.full((rows, D), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    bd.qkv_norm_rope_fwd(G.dev(x), *[G.dev(w) for w in ws], *outs, nh, hd, gain_q=G.dev(gq), gain_k=G.dev(gk),
                         cos=G.dev(cos, torch.float32), sin=G.dev(sin, torch.float32),
                         bq=G.dev(bs[0]), bk=G.dev(bs[1]), bv=G.dev(bs[2]))
    assert bd.device_status() == 0
    for i, gain in enumerate((gq, gk, None)):
        ref = oracle.linear(x, ws[i], bs[i])
        if gain is not None:
            ref = oracle.rope_apply(oracle.rms_norm_heads(ref, nh, hd, gain), nh, hd, cos, sin)
        G.check(G.host(outs[i]), ref, max_abs=2.0 ** -8 * np.abs(ref).max() + 1e-4, what=f"projection {i}")


# Map blocks: rows and keys around the 128 x 64 tiles, blocks that begin inside a segment
# and span two, heads that do not divide by the cluster, narrow heads.
@pytest.mark.parametrize("hd,nh,L,split,row0,rows,cols", [
    (128, 3, 200, 70, 33, 167, 150), (128, 24, 140, 12, 12, 128, 64), (64, 5, 300, 129, 0, 300, 65),
    (40, 8, 130, 1, 1, 129, 130), (128, 1, 129, 128, 128, 1, 1)])
def test_map_block_edges(bd, oracle, hd, nh, L, split, row0, rows, cols):
    q, k, v = _acts([(L, nh * hd)] * 3, 9900 + L, "bf16")
    bias = synth.normal((rows, cols), 9901, 0, 0.5)
    tq, tk, tv = G.dev(q), G.dev(k), G.dev(v)
    out = torch.empty_like(tq)
    seg = lambda t: [t[:split], t[split:]]
    amap = bd.sdpa_traced_fwd(seg(tq), seg(tk), seg(tv), seg(out), nh, bias=G.dev(bias, torch.float32),
                              bias_row0=row0, map_row0=row0, map_rows=rows, map_cols=cols)
    assert bd.device_status() == 0
    _, ref = oracle.sdpa(q, k, v, nh, bias=bias, bias_row0=row0, want_avg=True)
    # FP32 scores on both sides; 2^-22 from each exponential and 1e-5 from the sums
    assert np.abs(G.host(amap) - ref[row0:row0 + rows, :cols]).max() <= 1e-4 * ref.max()


# Key masks that leave whole key tiles out: the first, the last, all but one, every one, more
# tiles than the list of visible tiles holds.
@pytest.mark.parametrize("hd,Lk,first,last", [(128, 700, 300, 700), (128, 700, 0, 100), (64, 1000, 390, 395),
                                              (128, 300, 0, 0), (64, 512 * 128 + 77, 65000, 65600)])
def test_key_tiles_without_a_visible_key(bd, oracle, hd, Lk, first, last):
    nh, Lq = 2, 150
    q, k, v = _acts([(Lq, nh * hd), (Lk, nh * hd), (Lk, nh * hd)], 9560 + Lk, "bf16")
    mask = np.zeros(Lk, np.float32)
    mask[first:last] = 1.0
    got = G.sdpa(bd, q, k, v, nh, key_mask=mask)
    if last == first:
        assert not got.any()
        return
    ref = oracle.sdpa(q, k[first:last], v[first:last], nh)
    # probabilities are rounded to BF16 (2^-9 of each), then the output
    assert np.abs(got - ref).max() <= 2.0 ** -7 * np.abs(ref).max()


# Query tiles all of whose keys are masked (a left-padded prompt under the causal rule, a mask without a
# visible key): their rows are zero however late the query tile arrives.  Enough CTAs to fill the SMs,
# queries that come from HBM (L2 is flushed), several repeats.
@pytest.mark.parametrize("hd,nh", [(128, 24), (64, 24), (40, 8)])
@pytest.mark.parametrize("masked,causal", [(300, True), (700, False)])
def test_query_tiles_without_a_visible_key(bd, oracle, hd, nh, masked, causal):
    B, L = 3, 700
    q, k, v = (synth.activations((B, L, nh * hd), 9580 + i) for i in range(3))
    mask = np.ones(L, np.float32)
    mask[:masked] = 0.0
    tq, tk, tv, tm = G.dev(q), G.dev(k), G.dev(v), G.dev(mask, torch.float32)
    flush = torch.empty(256 << 20, device="cuda", dtype=torch.uint8)
    first = None
    for _ in range(8):
        out = torch.full_like(tq, float("nan"))
        flush.fill_(1)
        bd.sdpa_fwd(tq, tk, tv, out, nh, key_mask=tm, mask_mode=bd.MASK_CAUSAL if causal else bd.MASK_NONE)
        assert bd.device_status() == 0
        assert not out[:, :masked].any()
        first = out if first is None else first
        assert torch.equal(out, first)
    if masked < L:
        ref = oracle.sdpa(q[1, masked:], k[1, masked:], v[1, masked:], nh, mask_mode=1)
        # probabilities are rounded to BF16 (2^-9 of each), then the output
        assert np.abs(G.host(first[1, masked:]) - ref).max() <= 2.0 ** -7 * np.abs(ref).max()


def test_a_refused_launch_leaves_the_next_call_alone(bd):
    """More heads than a grid has rows is refused, and the next call does not report that error again."""
    x = torch.zeros(1, 65536 * 136, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(bd.BdattnError, match=r"^bdattn_sdpa_fwd: CUDA error"):
        bd.sdpa_fwd(x, x, x, torch.empty_like(x), 65536)
    t = torch.ones(4, 256, device="cuda", dtype=torch.bfloat16)
    cos, sin = torch.ones(4, 64, device="cuda"), torch.zeros(4, 64, device="cuda")
    out = torch.empty_like(t)
    bd.rmsnorm_rope([dict(x=t, out=out, cos=cos, sin=sin)], 2, 128, pair_mode=1)
    assert torch.equal(out, t)
