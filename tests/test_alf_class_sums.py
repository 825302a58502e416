"""Luma ALF classes of blocks whose gradient sums are as large as samples allow:
stripes and checkers of 4095 and of samples above the bit depth, in the chain and
in the encoder's trials."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import abi, native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu

PATTERNS = {"columns": lambda y, x: x & 1, "rows": lambda y, x: y & 1, "checker": lambda y, x: (x + y) & 1,
            "diagonal": lambda y, x: (x + y) >> 1 & 1}


def picture(bd, value, pattern):
    pic, fa = W.make_workload(60 + bd, 200, 136, bd, 6, ccalf=True, n_luma_aps=2, n_chroma_alt=2)
    fa.deblock.disabled = 1
    fa.sao[:] = np.zeros_like(fa.sao)  # the samples reach ALF as they are
    y, x = np.mgrid[0:104, 0:150]
    pic.luma[16:120, 20:170] = np.where(PATTERNS[pattern](y, x), value, 0)
    return pic, fa


@pytest.mark.parametrize("bd,value", [(8, 8000), (8, 16383), (10, 4095), (10, 8000), (10, 16383), (12, 4095),
                                      (12, 4096), (12, 16383), (13, 8191), (14, 16383)])
@pytest.mark.parametrize("pattern", sorted(PATTERNS))
def test_chain(bd, value, pattern):
    pic, fa = picture(bd, value, pattern)
    want = pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    with native.Context(0) as ctx:
        got = pic.copy()
        ctx.apply_in_loop_filters(got, fa)
        plan, dev = ctx.plan(pic, fa), native.DevicePicture.from_host(pic)
        ctx.execute_plans([plan], [dev])
        ctx.synchronize()
        assert dev.to_host().equal(want)
    assert got.equal(want)


@pytest.mark.parametrize("bd,value", [(8, 8000), (10, 8000), (12, 4096), (12, 16383), (14, 16383)])
@pytest.mark.parametrize("pattern", sorted(PATTERNS))
def test_trials(bd, value, pattern):
    rec, fa = picture(bd, value, pattern)
    src = rec.copy()
    oracle.apply_alf_clipped(src, fa)  # an original that the filters come near to
    want, got = rec.copy(), rec.copy()
    kw = dict(ctb_log2=6, bit_depth=bd)
    dw, sw = oracle.alf_decide_and_apply(src, want, fa.apses[0], alf_ctb_dtype=abi.ALF_CTB, **kw)
    with native.Context(0) as ctx:
        dg, sg = native.alf_decide_and_apply(ctx, src, got, fa.apses[0], want_sse=True, **kw)
    assert np.array_equal(sw, sg)
    assert dw.tobytes() == dg.tobytes()
    assert got.equal(want)
