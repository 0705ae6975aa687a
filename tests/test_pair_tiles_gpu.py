"""Linear layers on CTA pairs with both tile widths, 256 and 128 accumulator columns (csrc/gemm_plan.h chooses):
ragged rows and K, one tile and several to a pair, two heads, one head and half a head of 128 to an epilogue
warp.  Bounds: one rounding to the storage type of values of up to about five, as in test_qkv_proj_gpu.py, and the
reference's for GEGLU (tests/test_fused_parity.cpp:168-239)."""
import numpy as np
import pytest
import torch

import gpu_util as G
import synth

pytestmark = pytest.mark.gpu

TYPES = {"bf16": (torch.bfloat16, synth.round_bf16), "fp16": (torch.float16, synth.round_fp16)}


@pytest.mark.parametrize("storage", ["bf16", "fp16"])
@pytest.mark.parametrize("rows,din,nh,hd", [
    (509, 1000, 24, 128), (509, 1000, 48, 64),       # 256 columns, one tile to a pair
    (1000, 1000, 24, 128),                           # 256 columns, two tiles
    (129, 200, 3, 128), (77, 72, 6, 64),             # 128 columns, no multiple of 256
    (1500, 72, 8, 128)])                             # 128 columns, two tiles
def test_heads(bd, oracle, storage, rows, din, nh, hd):
    dt, rnd = TYPES[storage]
    D = nh * hd
    x = rnd(synth.normal((rows, din), 9700 + rows, 0, 1.0))
    ws = [rnd(synth.normal((D, din), 9701 + rows + i, 0, 1.0 / din ** 0.5)) for i in range(3)]
    bs = [rnd(synth.normal((D,), 9705 + rows + i, 0, 0.1)) for i in range(3)]
    gs = [synth.gains(hd, 9710 + i, "f32") for i in range(2)]
    cos, sin = oracle.flux_rope_tables(100, 40, 40, hd, (16, 56, 56) if hd == 128 else (8, 28, 28))
    outs = [torch.full((rows, D), float("nan"), device="cuda", dtype=dt) for _ in range(3)]
    bd.qkv_norm_rope_fwd(G.dev(x, dt), *[G.dev(w, dt) for w in ws], *outs, nh, hd,
                         gain_q=G.dev(gs[0], torch.float32), gain_k=G.dev(gs[1], torch.float32),
                         cos=G.dev(cos, torch.float32), sin=G.dev(sin, torch.float32), rope_row0=5,
                         bq=G.dev(bs[0], dt), bk=G.dev(bs[1], dt), bv=G.dev(bs[2], dt))
    assert bd.device_status() == 0
    for i in range(3):
        ref = oracle.linear(x, ws[i], bs[i])
        if i < 2:
            ref = oracle.rope_apply(oracle.rms_norm_heads(ref, nh, hd, gs[i]), nh, hd, cos[5:], sin[5:])
        assert np.abs(G.host(outs[i]) - ref).max() < 2.5e-2


@pytest.mark.parametrize("M,N,K", [(1100, 2176, 200), (2100, 1152, 72)])
def test_linear_128_columns(bd, oracle, M, N, K):
    x, w = synth.activations((M, K), 9800), synth.round_bf16(synth.normal((N, K), 9801, 0, 1.0 / K ** 0.5))
    b = synth.weights((N,), 9802)
    y = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    bd.linear_fwd(G.dev(x), G.dev(w), G.dev(b), y)
    assert bd.device_status() == 0
    G.check(G.host(y), oracle.linear(x, w, b), max_abs=2.5e-2, what=f"linear {M}x{N}x{K}")


@pytest.mark.parametrize("B,Din,Dout", [(130, 520, 192), (1, 64, 64), (1000, 616, 2560)])
def test_geglu_64_columns(bd, oracle, B, Din, Dout):
    x = synth.activations((B, Din), 9900 + B, "fp16")
    w = synth.round_fp16(synth.normal((2 * Dout, Din), 9901 + B, 0, 1.0 / Din ** 0.5))
    b = synth.round_fp16(synth.normal((2 * Dout,), 9902 + B, 0, 0.2))
    y = torch.full((B, Dout), float("nan"), device="cuda", dtype=torch.float16)
    bd.linear_geglu_fwd(G.dev(x, torch.float16), G.dev(w, torch.float16), G.dev(b, torch.float16), y)
    assert bd.device_status() == 0
    ref = oracle.linear_geglu(x, w, b)
    got = G.host(y)
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= 0.01 * np.abs(ref).max() + 0.008


@pytest.mark.parametrize("M,N,K", [(1100, 2176, 712), (577, 4992, 456),           # 128 columns
                                   (1000, 3072, 616), (999, 3072, 1000)])         # 256 columns
def test_linear_both_widths(bd, oracle, M, N, K):
    """Plain layers on pairs (tests/test_gemm_plan.py has the width of each), ragged rows and K."""
    x, w = synth.activations((M, K), 9740), synth.round_bf16(synth.normal((N, K), 9741, 0, 1.0 / K ** 0.5))
    b = synth.weights((N,), 9742)
    y = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    bd.linear_fwd(G.dev(x), G.dev(w), G.dev(b), y[:M, :N])
    assert bd.device_status() == 0
    G.check(G.host(y[:M, :N]), oracle.linear(x, w, b), max_abs=2.5e-2, what=f"linear {M}x{N}x{K}")
    assert bool((y[M] == 7.0).all()) and bool((y[:, N:] == 7.0).all())
