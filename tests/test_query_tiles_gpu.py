"""CTAs with two query tiles against CTAs with one, bit for bit, over the options of an attention call.

A launch whose pairs of query tiles fill no more than half of the SMs runs single tiles, which is what the tests
against the oracle are, being small.  Here a call of many heads runs pairs, or pairs and single tiles, and the
same heads three at a time run single tiles (148 SMs); a row's arithmetic is the same in all."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows of two query segments, batch items, heads: 120 pairs of tiles; 192 pairs of which the last 44 run as single tiles
WAVES = {"pairs": ([600, 400], 1, 24), "both": ([300, 1400], 1, 24), "both, two items": ([300, 1400], 2, 12)}
KINDS = ["plain", "q_norm", "q_norm causal", "grouped", "grouped q_norm masked", "all masked", "masked scaled", "causal masked"]


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("wave", list(WAVES))
@pytest.mark.parametrize("kind", KINDS)
def test_pairs_have_the_bits_of_single_tiles(bd, kind, wave, hd):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the wave sizes are those of 148 SMs")
    rows, B, nh = WAVES[wave]
    Lk, group = 700, 3 if "grouped" in kind else 1
    if "q_norm" in kind and B > 1:
        pytest.skip("one batch item")
    gen = torch.Generator(device="cuda").manual_seed(9300 + hd)
    rnd = lambda n, heads, dt=torch.bfloat16: torch.randn(B, n, heads * hd, device="cuda", generator=gen).to(dt)
    q, k, v = [rnd(n, nh) for n in rows], rnd(Lk, nh // group), rnd(Lk, nh // group)
    kw = {}
    if "q_norm" in kind:
        f = lambda *s: torch.randn(*s, device="cuda", generator=gen)
        kw["q_norm"] = dict(gain=[1 + 0.1 * f(hd), 1 + 0.1 * f(hd)], cos=f(sum(rows) + 3, hd // 2), sin=f(sum(rows) + 3, hd // 2), rope_row0=3)
    if "causal" in kind:
        kw["mask_mode"] = bd.MASK_CAUSAL            # more queries than keys: the first rows see none
    if "masked" in kind:
        kw["key_mask"] = (torch.rand(Lk, device="cuda", generator=gen) > 0.4).float()
        kw["key_mask"][128:384] = 0.0
        if "all" in kind:
            kw["key_mask"].zero_()
    if "scaled" in kind:
        kw["key_scale"] = 0.5 + torch.rand(Lk, device="cuda", generator=gen)
        kw["val_scale"] = 0.5 + torch.rand(Lk, device="cuda", generator=gen)
    out, ref = [torch.full_like(x, float("nan")) for x in q], [torch.full_like(x, float("nan")) for x in q]
    bd.sdpa_fwd(q, k, v, out, nh, num_kv_heads=nh // group, **kw)
    for b in range(B):
        for h in range(0, nh, 3):
            c, kc = slice(h * hd, (h + 3) * hd), slice(h // group * hd, (h // group + 3 // group) * hd)
            bd.sdpa_fwd([x[b:b + 1, :, c] for x in q], k[b:b + 1, :, kc], v[b:b + 1, :, kc], [x[b:b + 1, :, c] for x in ref], 3,
                        num_kv_heads=3 // group, **kw)
    assert bd.device_status() == 0
    for a, r in zip(out, ref):
        assert torch.equal(a, r)
    if "all" in kind:
        assert not any(bool(x.any()) for x in out)
