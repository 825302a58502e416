"""The packed SAO / ALF tile pass at the edges of its forms: windows by quads
of samples (picture widths that leave partial quads, clip rectangles at tile
borders, neighbouring CTBs of every SAO type), the offset form of the clipped
taps at every bit depth it takes, and tiles with samples outside the bit depth,
which take the plain form."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [(64, 64, 6), (68, 66, 6), (130, 70, 6), (134, 134, 7), (198, 66, 5), (258, 130, 7)]


def check(pic, fa, what):
    want = pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    with native.Context(0) as ctx:
        got = pic.copy()
        ctx.apply_in_loop_filters(got, fa)
        assert got.equal(want), f"{what}: one picture"
        for tile_h in (64, 32):
            ctx.set_tuning("sao_alf_tile_h", tile_h)
            plans, devs = [ctx.plan(pic, fa)], [native.DevicePicture.from_host(pic)]
            ctx.execute_plans(plans, devs)
            ctx.synchronize()
            assert devs[0].to_host().equal(want), f"{what}: batch, tile height {tile_h}"


@pytest.mark.parametrize("w,h,log2", SIZES)
@pytest.mark.parametrize("bd", [8, 10, 12, 14])
def test_sizes_and_depths(w, h, log2, bd):
    pic, fa = W.make_workload(100 * bd + w, w, h, bd, log2, ccalf=True, lmcs=bd <= 12, n_luma_aps=2, n_chroma_alt=2,
                              alf_fixed_frac=0.3)
    check(pic, fa, f"{w}x{h} {bd} bit CTB {1 << log2}")


@pytest.mark.parametrize("bd", [8, 10, 13])
def test_tiles_at_clip_rectangles(bd):
    pic, fa = W.make_workload(77, 390, 262, bd, 6, ccalf=True, tiles=([2, 1, 3, 1], [2, 3]))
    check(pic, fa, f"tiles, {bd} bit")


@pytest.mark.parametrize("bd,value", [(10, 16383), (10, 16384), (12, 20000), (14, 16384), (14, 30000)])
def test_samples_outside_the_depth(bd, value):
    """Samples no decoder produces, in some tiles only: SAO off for them to reach ALF as they are."""
    pic, fa = W.make_workload(88 + bd, 200, 136, bd, 6, ccalf=True, n_luma_aps=2, n_chroma_alt=2)
    fa.deblock.disabled = 1
    fa.sao[:] = np.zeros_like(fa.sao)
    rng = np.random.default_rng(bd)
    for p in pic.planes():
        p[rng.integers(0, p.shape[0] // 2, 20), rng.integers(0, p.shape[1] // 2, 20)] = value
    check(pic, fa, f"{bd} bit with samples of {value}")


@pytest.mark.parametrize("tile_h,cps", [(64, 0), (32, 0), (64, 2)])
def test_large_tiles_in_a_batch(tile_h, cps):
    """The same sizes and depths in one batch with more 64 x 64 tiles than SMs, which keeps the large tiles."""
    items = [W.make_workload(100 * bd + w, w, h, bd, log2, ccalf=True, lmcs=bd <= 12, n_luma_aps=2, n_chroma_alt=2,
                             alf_fixed_frac=0.3) for bd in (8, 10, 12, 14) for w, h, log2 in SIZES]
    items += [W.make_workload(5, 832, 480, 10, 7, ccalf=True)]
    with native.Context(0) as ctx:
        ctx.set_tuning("sao_alf_tile_h", tile_h)
        ctx.set_tuning("sao_alf_ctas_per_sm", cps)
        plans = [ctx.plan(p, f) for p, f in items]
        devs = [native.DevicePicture.from_host(p) for p, _ in items]
        ctx.execute_plans(plans, devs)
        ctx.synchronize()
    for (p, f), d in zip(items, devs):
        want = p.copy()
        oracle.apply_in_loop_filters(want, f)
        assert d.to_host().equal(want), (p.width, p.height, p.bit_depth)
