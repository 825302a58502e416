"""SAO, ALF and CC-ALF of 4:2:2 and 4:4:4 in the packed tiles: planes that end
inside a tile or a run of four, every CTB size (4:2:2 at CTB 32 has its own tile
width), clip rectangles, depths up to 14 bits, and a batch of all of them."""
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = [(64, 64, 5, 8, 2), (68, 36, 5, 10, 2), (134, 70, 6, 12, 2), (258, 130, 7, 10, 2), (66, 40, 5, 10, 3),
         (130, 66, 6, 14, 3), (200, 136, 7, 8, 3), (262, 134, 7, 12, 3)]


def make(w, h, log2, bd, cfi):
    tiles = ([1, 1, -(-w // (1 << log2)) - 2], [-(-h // (1 << log2))]) if w > 3 << log2 else None
    pic, fa = W.make_workload(60 * w + bd, w, h, bd, log2, inter_frac=0.3, ccalf=True, lmcs=bd <= 12, n_luma_aps=2,
                              n_chroma_alt=3, tiles=tiles)
    return W.with_chroma_format(pic, fa, cfi, w)


@pytest.mark.parametrize("case", CASES)
def test_single(case):
    pic, fa = make(*case)
    want = pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    with native.Context(0) as ctx:
        got = pic.copy()
        ctx.apply_in_loop_filters(got, fa)
        assert got.equal(want)
        for name in ("sao", "alf"):
            got, want = pic.copy(), pic.copy()
            getattr(ctx, f"apply_{name}_clipped")(got, fa)
            getattr(oracle, f"apply_{name}_clipped")(want, fa)
            assert got.equal(want), name


def test_batch():
    items = [make(*c) for c in CASES] + [W.config1(5)]
    with native.Context(0) as ctx:
        plans = [ctx.plan(p, f) for p, f in items]
        devs = [native.DevicePicture.from_host(p) for p, _ in items]
        ctx.execute_plans(plans, devs)
        ctx.synchronize()
    for (p, f), d, c in zip(items, devs, CASES + ["4:2:0"]):
        want = p.copy()
        oracle.apply_in_loop_filters(want, f)
        assert d.to_host().equal(want), c
