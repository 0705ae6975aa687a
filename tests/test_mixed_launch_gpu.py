"""A launch of the one-tile linear kernel that mixes a projection with per-head RMSNorm and one without
(tests/cpp/mixed_launch.cu): each gets its own epilogue, the plain one its bias."""
import ctypes as C
import os
import subprocess

import pytest
import torch

import gpu_util as G
import synth

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "cpp", "mixed_launch.so")


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,n1,bias", [(200, 256, 136, True), (64, 72, 64, True), (300, 640, 192, False)])
def test_norm_and_plain_projection_in_one_launch(bd, oracle, M, K, n1, bias):
    src = [os.path.join(HERE, "cpp", "mixed_launch.cu")]
    src += [os.path.join(HERE, "..", "brodiffusion_b200", "csrc", n) for n in ("gemm_tc05.cu", "tc05.cuh", "gemm_plan.h", "sdpa_internal.h")]
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(map(os.path.getmtime, src)):
        subprocess.check_call(["sh", os.path.join(HERE, "cpp", "build.sh")])
    run = C.CDLL(LIB).mixed_launch
    p, i, f = C.c_void_p, C.c_int, C.c_float
    run.argtypes = [p, i, i, p, i, p, f, p, p, i, p, p]
    x = synth.activations((M, K), 9970)
    w0, w1 = (synth.round_bf16(synth.normal((n, K), 9971 + n, 0, 1.0 / K ** 0.5)) for n in (192, n1))
    b, gain = synth.round_bf16(synth.normal((n1,), 9973, 0, 1.0)), synth.gains(64, 9974, "f32")
    tx, t0, t1, tb, tg = G.dev(x), G.dev(w0), G.dev(w1), G.dev(b), G.dev(gain, torch.float32)
    y0, y1 = (torch.full((M, n), float("nan"), device="cuda", dtype=torch.bfloat16) for n in (192, n1))
    torch.cuda.synchronize()
    assert run(tx.data_ptr(), M, K, t0.data_ptr(), 192, tg.data_ptr(), 1e-6, y0.data_ptr(), t1.data_ptr(), n1,
               tb.data_ptr() if bias else None, y1.data_ptr()) == 0
    # bounds: one rounding to BF16 of values of up to about five
    G.check(G.host(y0), oracle.rms_norm_heads(oracle.linear(x, w0, None), 3, 64, gain), max_abs=2.5e-2, what="norm")
    G.check(G.host(y1), oracle.linear(x, w1, b if bias else None), max_abs=2.5e-2, what="plain")
