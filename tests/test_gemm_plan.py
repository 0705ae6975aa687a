"""The rule that chooses kernel, tile width and split of a launch of linear layers, on the
CPU: csrc/gemm_plan.h is plain C++ and is compiled here into a small library."""
import ctypes as C
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plan") / "plan.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", so,
                           os.path.join(ROOT, "tests", "cpp", "gemm_plan_probe.cpp")])
    lib = C.CDLL(so)

    def run(shapes, geglu=False, heads=False, sms=148):
        flat = (C.c_int * (3 * len(shapes)))(*itertools.chain(*shapes))
        out = (C.c_int * 4)()
        lib.probe_plan(flat, len(shapes), int(geglu), int(heads), sms, out)
        run.pair_cols = out[3]
        return bool(out[0]), out[1], out[2]

    def kernel(shapes, **kw):
        """Name of the kernel and tile width, and over how many CTAs a tile is split."""
        pair, width, split = run(shapes, **kw)
        return f"p{run.pair_cols}" if pair else str(width), split

    run.kernel = kernel
    run.fewest_blocks = lib.probe_fewest_blocks
    run.acc_reused = lib.probe_acc_reused
    return run


def test_every_cta_of_a_split_tile_has_a_k_block(plan):
    """Q, K and V of a cross-attention in one launch: K is x_cols for Q and ctx_cols for the others."""
    splits = set()
    for rows, ctx_rows, inner, x_cols, ctx_cols in itertools.product(
            (1, 64, 256, 1000, 4096), (16, 77, 256, 512), (64, 128, 192, 256, 320, 640, 768, 1280, 3072),
            (8, 64, 128, 192, 320, 640, 1280), (8, 64, 128, 320, 768, 1024, 2048, 4096)):
        shapes = [(rows, inner, x_cols), (ctx_rows, inner, ctx_cols), (ctx_rows, inner, ctx_cols)]
        pair, width, split = plan(shapes)
        splits.add(split)
        assert not (pair and split > 1)
        for _, _, k in shapes:
            assert plan.fewest_blocks(k, split) >= 1, (shapes, split)
    assert splits == {1, 2, 4, 8}


@pytest.mark.parametrize("shapes,split", [
    ([(64, 64, 64), (77, 64, 768), (77, 64, 768)], 1),
    ([(64, 192, 192), (77, 192, 768), (77, 192, 768)], 2),
    ([(256, 256, 256), (77, 256, 2048), (77, 256, 2048)], 4),
    ([(64, 1280, 1280), (77, 1280, 64), (77, 1280, 64)], 1),
    ([(64, 1280, 5120)], 8), ([(256, 1280, 1280)], 2), ([(128, 64, 768)], 4), ([(128, 64, 704)], 2),
    ([(128, 64, 640)], 1)])
def test_split_is_bounded_by_the_shortest_k(plan, shapes, split):
    assert plan(shapes)[2] == split


# kernel (64 to 128: columns of the one-tile kernel; p128, p256: pairs) that the measurements beside the rule have as
# the fastest or within 3 % of it: short K, where a pair waits for its epilogues; long K; rows off 32 bytes
@pytest.mark.parametrize("kind,shape,kernels", [
    ("plain", (2304, 2560, 320), ("80", "112", "128")), ("plain", (4096, 1280, 320), ("80", "112", "128")),
    ("plain", (9216, 640, 320), ("80", "112", "128")), ("plain", (4096, 2560, 112), ("96", "128")),
    ("plain", (9216, 1280, 640), ("p256",)), ("plain", (2240, 2304, 2240), ("p128",)),
    ("plain", (576, 5120, 448), ("96", "p128")), ("plain", (576, 4096, 936), ("p256",)), ("plain", (2240, 1024, 2240), ("128",)),
    ("geglu", (4096, 1280, 2808), ("p256",)), ("geglu", (64, 5120, 1280), ("p128",)), ("geglu", (4096, 1280, 320), ("p256",)),
    ("heads", (3580, 1024, 1288), ("p256",)), ("heads", (256, 3072, 3072), ("p128",)), ("heads", (1024, 3072, 3072), ("p256",))])
def test_plan_is_the_measured_best(plan, kind, shape, kernels):
    n = 3 if kind == "heads" else 1
    assert plan.kernel([shape] * n, geglu=kind == "geglu", heads=kind == "heads")[0] in kernels


def test_geglu_is_never_split(plan):
    for rows, d_in, d_out in itertools.product((1, 64, 300, 4096), (64, 320, 1280, 5120), (72, 128, 1280, 5120)):
        assert plan([(rows, d_out, d_in)], geglu=True)[2] == 1


@pytest.mark.parametrize("pairs", [1, 2, 74])
@pytest.mark.parametrize("total", [1, 2, 3, 4, 5, 73, 74, 75, 147, 148, 149, 222, 223, 1000])
def test_every_release_of_an_accumulator_is_waited_for(plan, pairs, total):
    """The MMA issuer of a pair waits, before its tile ti >= 2, for the release of tile ti - 2.  A release
    that it does not wait for could reach a CTA that has ended."""
    for first in range(min(pairs, total)):
        tiles = list(range(first, total, pairs))
        released = [ti for ti, tile in enumerate(tiles) if plan.acc_reused(tile, pairs, total)]
        assert released == [ti - 2 for ti in range(2, len(tiles))]


@pytest.mark.parametrize("shape", [(65, 1280, 5120), (100, 1280, 5120), (135, 640, 5120), (131, 608, 4736), (223, 1264, 2640)])
def test_no_split_beyond_the_sms_above_64_rows(plan, shape):
    """Where the parts do not all run at once the exchange of full tiles costs more than the shorter K saves."""
    m, n, _ = shape
    assert -(-m // 128) * -(-n // 64) * plan([shape])[2] <= 148


@pytest.mark.parametrize("shape,kernels", [
    ((3829, 5016, 392), ("128",)), ((8128, 1696, 504), ("128",)), ((2341, 3320, 280), ("128",)), ((2079, 4608, 392), ("p256",)),
    ((1895, 1184, 136), ("64",)), ((7290, 392, 216), ("64", "96")), ((2569, 1288, 248), ("64", "96")), ((1911, 2112, 200), ("64", "96")),
    ((8256, 2848, 1208), ("80", "128")), ((4399, 3768, 1032), ("80", "128")), ((8218, 1728, 1032), ("80", "128"))])
def test_k_off_32_bytes(plan, shape, kernels):
    """More tiles than SMs: a width that was measured to be no slower than 128 columns were before the pair kernel's narrow tiles."""
    assert plan.kernel([shape])[0] in kernels


# What the GPU tests of single kernels say that they run (148 SMs): a change of the modelled times must not empty them
@pytest.mark.parametrize("kind,shapes,kernel", [
    ("heads", [(509, 3072, 1000), (1000, 3072, 1000)], "p256"), ("heads", [(129, 384, 200), (77, 384, 72), (1500, 1024, 72)], "p128"),
    ("geglu", [(130, 192, 520), (1, 64, 64), (1000, 2560, 616), (2300, 1152, 200)], "p128"), ("geglu", [(4096, 1280, 320)], "p256"),
    ("plain", [(1100, 2176, 712), (577, 4992, 456)], "p128"), ("plain", [(1000, 3072, 616), (999, 3072, 1000)], "p256"),
    ("plain", [(2300, 640, 640), (4000, 320, 72)], "80"), ("plain", [(500, 3072, 200)], "96"), ("plain", [(5000, 328, 600)], "112"),
    ("several", [(9200, 320, 648), (7000, 328, 648), (4800, 480, 1280), (7000, 328, 1288)], "80")])
def test_kernels_of_the_gpu_tests(plan, kind, shapes, kernel):
    for m, n, k in shapes:
        got = plan.kernel([(m, n, k)] * (3 if kind == "heads" else 1), geglu=kind == "geglu", heads=kind == "heads")
        assert got == (kernel, 1), (m, n, k)
        if kernel.isdigit():
            assert (-(-m // 128) * -(-n // int(kernel)) > 148) == (kind == "several")


@pytest.mark.parametrize("rows", [1, 64, 65, 128, 190])
@pytest.mark.parametrize("k,split", [(696, 2), (776, 4), (1544, 8)])
def test_splits_of_the_gpu_tests(plan, rows, k, split):
    for n in (8, 16, 24, 40, 64, 72, 104):
        assert plan([(rows, n, k)])[2] == split
