"""Traced / steered attention on the device against the oracle's statement of
dit::joint_attention_traced (src/dit/common.cpp:198-329): logit bias on the
image-query x text-key block and the head-averaged softmax block."""
import numpy as np
import pytest
import torch

import gpu_util as G
import synth

pytestmark = pytest.mark.gpu


def test_golden_flux_tiny_bias_and_map(bd, golden):
    g = golden
    nh, hd, txt = 2, 8, 3
    q, k, v = G.dev(g["flux_q"]), G.dev(g["flux_k"]), G.dev(g["flux_v"])
    cos, sin = G.dev(g["flux_cos"], torch.float32), G.dev(g["flux_sin"], torch.float32)
    qr, kr = torch.empty_like(q), torch.empty_like(k)
    bd.rmsnorm_rope([dict(x=q, out=qr, gain=G.dev(g["flux_gq"]), cos=cos, sin=sin),
                     dict(x=k, out=kr, gain=G.dev(g["flux_gk"]), cos=cos, sin=sin)], nh, hd)
    L = q.shape[0]
    out = torch.empty_like(q)
    amap = bd.sdpa_traced_fwd(qr, kr, v, out, nh, map_row0=0, map_rows=L, map_cols=L)
    assert bd.device_status() == 0
    G.check(G.host(out), g["flux_out"], what="traced output")
    assert np.abs(G.host(amap) - g["flux_avg"]).max() < 2e-2
    # rows of the full map are non-negative and sum to one (tests/test_flux_blocks.cpp:268-281)
    m = G.host(amap)
    assert m.min() >= 0.0 and np.abs(m.sum(1) - 1.0).max() < 2e-2
    outb = torch.empty_like(q)
    bd.sdpa_traced_fwd(qr, kr, v, outb, nh, bias=G.dev(g["flux_bias"], torch.float32), bias_row0=txt)
    assert bd.device_status() == 0
    G.check(G.host(outb), g["flux_out_biased"], what="biased output")


def test_flux_image_to_text_block(bd, oracle):
    """The block Flux keeps: image-query rows x text-key columns, with a bias that
    steers image tokens toward some text tokens (tests/test_flux_blocks.cpp:343-386)."""
    nh, hd, txt, img = 4, 128, 96, 400
    L, D = txt + img, nh * hd
    q, k, v = (synth.activations((L, D), 9100 + i) for i in range(3))
    bias = np.zeros((img, txt), np.float32)
    bias[:, 10:20] = 2.0
    tq, tk, tv = G.dev(q), G.dev(k), G.dev(v)
    out = torch.empty_like(tq)
    amap = bd.sdpa_traced_fwd([tq[:txt], tq[txt:]], [tk[:txt], tk[txt:]], [tv[:txt], tv[txt:]],
                              [out[:txt], out[txt:]], nh, bias=G.dev(bias, torch.float32), bias_row0=txt,
                              map_row0=txt, map_rows=img, map_cols=txt)
    assert bd.device_status() == 0
    ref_out, ref_avg = oracle.sdpa(q, k, v, nh, bias=bias, bias_row0=txt, want_avg=True)
    G.check(G.host(out), ref_out, what="steered output")
    got = G.host(amap)
    assert np.abs(got - ref_avg[txt:, :txt]).max() < 5e-3
    # steering is monotone: biased columns receive more weight than without bias
    amap0 = bd.sdpa_traced_fwd(tq, tk, tv, torch.empty_like(tq), nh, map_row0=txt, map_rows=img, map_cols=txt)
    assert G.host(amap)[:, 10:20].sum() > G.host(amap0)[:, 10:20].sum()


def test_unet_cross_attention_map(bd, oracle):
    """U-Net trace mode: map (Lq, 77) over all rows with a full (Lq, Lk) logit
    bias; rows sum to one within 0.05 (tests/test_unet.cpp:487-500)."""
    nh, hd, Lq, Lk = 8, 40, 256, 77
    q = synth.activations((Lq, nh * hd), 9201)
    k = synth.activations((Lk, nh * hd), 9202)
    v = synth.activations((Lk, nh * hd), 9203)
    bias = synth.normal((Lq, Lk), 9204, 0, 0.5)
    out = torch.empty(Lq, nh * hd, device="cuda", dtype=torch.bfloat16)
    amap = bd.sdpa_traced_fwd(G.dev(q), G.dev(k), G.dev(v), out, nh, bias=G.dev(bias, torch.float32),
                              map_rows=Lq, map_cols=Lk)
    assert bd.device_status() == 0
    ref_out, ref_avg = oracle.sdpa(q, k, v, nh, bias=bias, want_avg=True)
    G.check(G.host(out), ref_out, what="unet traced output")
    got = G.host(amap)
    assert np.abs(got - ref_avg).max() < 5e-3
    assert np.abs(got.sum(1) - 1.0).max() < 0.05


def test_map_agrees_with_masked_attention(bd, oracle):
    """The map block follows the visibility rules the attention itself used: a
    masked or future key has weight 0 and every visible row still sums to one."""
    nh, hd, Lq, Lk = 4, 64, 200, 200
    q, k, v = (synth.activations((Lq, nh * hd), 9300 + i) for i in range(3))
    tq, tk, tv = G.dev(q), G.dev(k), G.dev(v)
    # key mask (padded caption tail + a hole)
    mask = np.ones(Lk, np.float32)
    mask[150:] = 0.0
    mask[7] = 0.0
    out = torch.empty_like(tq)
    amap = bd.sdpa_traced_fwd(tq, tk, tv, out, nh, map_rows=Lq, map_cols=Lk, key_mask=G.dev(mask, torch.float32))
    assert bd.device_status() == 0
    ref_out, ref_avg = oracle.sdpa(q, k, v, nh, key_mask=mask, want_avg=True)
    G.check(G.host(out), ref_out, what="key-masked traced output")
    m = G.host(amap)
    assert np.abs(m - ref_avg).max() < 5e-3
    assert np.all(m[:, mask == 0.0] == 0.0)
    assert np.abs(m.sum(1) - 1.0).max() < 2e-2
    # causal
    out_c = torch.empty_like(tq)
    amap_c = bd.sdpa_traced_fwd(tq, tk, tv, out_c, nh, map_rows=Lq, map_cols=Lk, mask_mode=bd.MASK_CAUSAL)
    assert bd.device_status() == 0
    ref_out_c, ref_avg_c = oracle.sdpa(q, k, v, nh, mask_mode=1, want_avg=True)
    G.check(G.host(out_c), ref_out_c, what="causal traced output")
    mc = G.host(amap_c)
    assert np.abs(mc - ref_avg_c).max() < 5e-3
    assert np.all(np.triu(mc, 1) == 0.0)
    assert mc.max() <= 1.0 + 1e-3 and np.abs(mc.sum(1) - 1.0).max() < 2e-2


def test_errors(bd):
    q = torch.zeros(64, 256, device="cuda", dtype=torch.bfloat16)
    b = torch.zeros(100, 10, device="cuda")
    with pytest.raises(bd.BdattnError, match=r"^joint_attention_traced: bias block"):
        bd.sdpa_traced_fwd(q, q, q, q.clone(), 2, bias=b)


@pytest.mark.parametrize("hd,split,row0,rows,cols,offset,ld", [
    (128, 70, 75, 300, 200, 0, 200), (128, 256, 256, 250, 256, 4, 264),      # rows of 16-byte pieces
    (128, 70, 40, 170, 131, 0, 131), (64, 129, 1, 377, 130, 1, 200),         # rows and bases that are no multiple of them
    (40, 128, 128, 1, 1, 3, 8), (64, 300, 0, 506, 506, 2, 510)])
def test_bias_rows_of_any_alignment(bd, oracle, hd, split, row0, rows, cols, offset, ld):
    """The bias is copied in pieces of 32 rows x 32 columns: blocks that begin and end inside a piece, a tile and a
    segment, strides above the width, bases off a 16-byte boundary."""
    nh, L = 3, 506
    q, k, v = (synth.activations((L, nh * hd), 9950 + i) for i in range(3))
    wide = torch.full((rows, ld + offset), 1e30, device="cuda")              # what lies around it must not be read as bias
    bias = wide[:, offset:offset + cols]
    ref_bias = synth.normal((rows, cols), 9953, 0, 1.0)
    bias.copy_(G.dev(ref_bias, torch.float32))
    tq, tk, tv = G.dev(q), G.dev(k), G.dev(v)
    out = torch.full_like(tq, float("nan"))
    seg = lambda t: [t[:split], t[split:]]
    amap = bd.sdpa_traced_fwd(seg(tq), seg(tk), seg(tv), seg(out), nh, bias=bias, bias_row0=row0, map_row0=row0,
                              map_rows=rows, map_cols=cols)
    assert bd.device_status() == 0
    # (the oracle's bias reaches to the last query: rows without one are zero there)
    to_the_end = np.concatenate([ref_bias, np.zeros((L - row0 - rows, cols), np.float32)])
    ref, avg = oracle.sdpa(q, k, v, nh, bias=to_the_end, bias_row0=row0, want_avg=True)
    G.check(G.host(out), ref, what="biased output")
    # FP32 scores on both sides; 2^-22 from each exponential and 1e-5 from the sums
    assert np.abs(G.host(amap) - avg[row0:row0 + rows, :cols]).max() <= 1e-4 * avg.max()


# Two segments of query rows, 24 heads: 48 pairs of query tiles, all run as single tiles; 120, all pairs; 192, pairs and
# single tiles (148 SMs)
ROWS = {"single": [200, 100], "pairs": [600, 400], "both": [300, 1400]}


@pytest.mark.parametrize("hd", [128, 40])
@pytest.mark.parametrize("tiles", list(ROWS))
def test_hooks_without_an_effect_keep_the_bits(bd, tiles, hd):
    """Statistics, a mask of ones, scale vectors of ones and a bias of zeros, each alone and together: every combination
    has a kernel of its own, and all have the bits of the call without hooks."""
    nh, Lk = 24, 700
    gen = torch.Generator(device="cuda").manual_seed(9800 + hd)
    rnd = lambda n: torch.randn(n, nh * hd, device="cuda", generator=gen).to(torch.bfloat16)
    q, k, v = [rnd(n) for n in ROWS[tiles]], rnd(Lk), rnd(Lk)
    ref = [torch.full_like(x, float("nan")) for x in q]
    bd.sdpa_fwd(q, k, v, ref, nh)
    ones, Lq = torch.ones(Lk, device="cuda"), sum(ROWS[tiles])
    ws = torch.empty(8 * nh * Lq, device="cuda", dtype=torch.uint8)
    bias = torch.zeros(Lq, Lk, device="cuda")
    for hooks in range(1, 16):
        t = None
        if hooks & 3:                                        # statistics (a traced call), with a bias or without
            t = bd.TraceParams()
            t.workspace, t.workspace_bytes = ws.data_ptr(), ws.numel()
            if hooks & 2:
                t.bias, t.bias_rows, t.bias_cols, t.bias_ld = bias.data_ptr(), Lq, Lk, Lk
        kw = dict(key_mask=ones) if hooks & 4 else {}
        if hooks & 8:
            kw.update(key_scale=ones, val_scale=ones)
        out = [torch.full_like(x, float("nan")) for x in q]
        bd.sdpa_fwd(q, k, v, out, nh, _trace=t, **kw)
        assert bd.device_status() == 0
        for a, b in zip(out, ref):
            assert torch.equal(a, b), hooks


@pytest.mark.parametrize("hd", [128, 40])
@pytest.mark.parametrize("tiles", ["pairs", "both"])
@pytest.mark.parametrize("cols,row0,rows", [(1, 0, 5), (31, 3, 40), (33, 130, 200), (64, 255, 2), (97, 500, 400), (128, 290, 333),
                                            (131, 590, 60), (500, 700, 300)])
def test_biased_pairs_have_the_bits_of_single_tiles(bd, tiles, hd, cols, row0, rows):
    """A single query tile has all pieces of a key tile's bias in flight at once, a tile of a pair one after the other: a
    head's bits are the same, and the map is the mean of the maps of its parts."""
    nh, part, Lk = 24, 3, 600
    n_rows = ROWS[tiles]
    Lq = sum(n_rows)
    rows = min(rows, Lq - row0)
    gen = torch.Generator(device="cuda").manual_seed(9900 + cols)
    rnd = lambda n: torch.randn(n, nh * hd, device="cuda", generator=gen).to(torch.bfloat16)
    q, k, v = [rnd(n) for n in n_rows], rnd(Lk), rnd(Lk)
    kw = dict(bias=torch.randn(rows, cols, device="cuda", generator=gen), bias_row0=row0, map_row0=row0, map_rows=rows, map_cols=cols)
    out, ref = [torch.full_like(x, float("nan")) for x in q], [torch.full_like(x, float("nan")) for x in q]
    amap = bd.sdpa_traced_fwd(q, k, v, out, nh, **kw)
    mean = torch.zeros_like(amap)
    for h in range(0, nh, part):
        c = slice(h * hd, (h + part) * hd)
        mean += bd.sdpa_traced_fwd([x[:, c] for x in q], k[:, c], v[:, c], [x[:, c] for x in ref], part, **kw) * (part / nh)
    assert bd.device_status() == 0
    for a, b in zip(out, ref):
        assert torch.equal(a, b)
    # FP32 sums of the same terms in another order
    assert (amap - mean).abs().max() <= 1e-5 * mean.max()


def test_rows_without_a_bias_at_the_smallest_scale(bd):
    """The reciprocal of the softmax scale is beyond FP32; rows that have no bias must not notice."""
    nh, hd, L, rows, scale = 2, 64, 200, 40, 1e-39
    gen = torch.Generator(device="cuda").manual_seed(9950)
    q, k, v = (torch.randn(L, nh * hd, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(3))
    out, ref = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    bd.sdpa_fwd(q, k, v, ref, nh, softmax_scale=scale)
    bias = torch.randn(rows, 100, device="cuda", generator=gen)
    ws = torch.empty(8 * nh * L, device="cuda", dtype=torch.uint8)
    t = bd.TraceParams()
    t.workspace, t.workspace_bytes = ws.data_ptr(), ws.numel()
    t.bias, t.bias_row0, t.bias_rows, t.bias_cols, t.bias_ld = bias.data_ptr(), 10, rows, 100, 100
    bd.sdpa_fwd(q, k, v, out, nh, softmax_scale=scale, _trace=t)
    assert bd.device_status() == 0
    assert bool(torch.isfinite(ref).all())
    assert torch.equal(out[:10], ref[:10]) and torch.equal(out[10 + rows:], ref[10 + rows:])
