"""Linear layers on the one-tile kernel: tiles split over a cluster, and tiles of widths between 64 and 128."""
import pytest
import torch

import gpu_util as G
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(65, 72, 768), (127, 200, 1536), (200, 1280, 1288), (64, 136, 5120)])
def test_linear_split_rows_over_the_cluster(bd, oracle, M, N, K):
    """The rows of a split tile are dealt out to the CTAs of its cluster: ragged rows and columns, two to eight CTAs."""
    x, w = synth.activations((M, K), 9950), synth.round_bf16(synth.normal((N, K), 9951, 0, 1.0 / K ** 0.5))
    b = synth.weights((N,), 9952)
    y = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    bd.linear_fwd(G.dev(x), G.dev(w), G.dev(b), y[:M, :N])
    assert bd.device_status() == 0
    G.check(G.host(y[:M, :N]), oracle.linear(x, w, b), max_abs=2.5e-2, what=f"linear {M}x{N}x{K}")
    assert bool((y[M] == 7.0).all()) and bool((y[:, N:] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(2300, 640, 640), (4000, 320, 72), (500, 3072, 200), (5000, 328, 600), (1024, 648, 1288)])
def test_linear_tile_widths_between_64_and_128(bd, oracle, M, N, K):
    """Widths of 80, 96 and 112 columns (csrc/gemm_plan.h): no multiple of the epilogue's 32, ragged rows, columns and
    K, one CTA to an SM and two.  Bound as in test_qkv_proj_gpu.py: one rounding of values of up to five."""
    x, w = synth.activations((M, K), 9960), synth.round_bf16(synth.normal((N, K), 9961, 0, 1.0 / K ** 0.5))
    b = synth.weights((N,), 9962)
    y = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    bd.linear_fwd(G.dev(x), G.dev(w), G.dev(b), y[:M, :N])
    assert bd.device_status() == 0
    G.check(G.host(y[:M, :N]), oracle.linear(x, w, b), max_abs=2.5e-2, what=f"linear {M}x{N}x{K}")
    assert bool((y[M] == 7.0).all()) and bool((y[:, N:] == 7.0).all())


@pytest.mark.parametrize("N", [8, 16, 24, 40, 64, 72, 104])
@pytest.mark.parametrize("M", [1, 64, 65, 128, 190])
def test_linear_split_shares_of_narrow_and_ragged_tiles(bd, oracle, M, N):
    """Tiles of one to eight pieces of eight columns; up to 64 rows, more, all: how a cluster shares the rows and a
    warp the pieces depends on both. The K give two, four and eight CTAs to a tile.  Bound as above."""
    for K in (696, 776, 1544):
        x, w = synth.activations((M, K), 9980), synth.round_bf16(synth.normal((N, K), 9981, 0, 1.0 / K ** 0.5))
        b = synth.weights((N,), 9982)
        y = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
        bd.linear_fwd(G.dev(x), G.dev(w), G.dev(b), y[:M, :N])
        assert bd.device_status() == 0
        G.check(G.host(y[:M, :N]), oracle.linear(x, w, b), max_abs=2.5e-2, what=f"linear {M}x{N}x{K}")
        assert bool((y[M] == 7.0).all()) and bool((y[:, N:] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(9200, 320, 648), (7000, 328, 648), (4800, 480, 1280), (7000, 328, 1288)])
def test_linear_80_columns_several_ctas_to_an_sm(bd, oracle, M, N, K):
    """80 columns with more tiles than SMs, where a ring of four stages lets two CTAs share one (tests/test_gemm_plan.py
    has the width of each).  Bound as above."""
    x, w = synth.activations((M, K), 9990), synth.round_bf16(synth.normal((N, K), 9991, 0, 1.0 / K ** 0.5))
    b = synth.weights((N,), 9992)
    y = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    bd.linear_fwd(G.dev(x), G.dev(w), G.dev(b), y[:M, :N])
    assert bd.device_status() == 0
    G.check(G.host(y[:M, :N]), oracle.linear(x, w, b), max_abs=2.5e-2, what=f"linear {M}x{N}x{K}")
    assert bool((y[M] == 7.0).all()) and bool((y[:, N:] == 7.0).all())
