"""Calls whose shape decides the route: map blocks at the edges of their tiles and
segments.  References: the CPU oracle."""
import numpy as np
import pytest
import torch

import gpu_util as G
import synth

pytestmark = pytest.mark.gpu


def _acts(shapes, seed, storage):
    return [synth.activations(s, seed + i, storage) for i, s in enumerate(shapes)]


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
