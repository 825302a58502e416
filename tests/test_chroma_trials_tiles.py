"""The encoder's chroma ALF and CC-ALF decisions at the edges of their tiles:
CTBs of 32, 64 and 128, chroma planes that end inside a tile, a run of four
samples or a pair, clip rectangles, and depths up to 14 bits."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import abi, native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,log2,bd", [(64, 64, 5, 8), (66, 34, 5, 10), (130, 70, 6, 10), (258, 134, 7, 12),
                                         (200, 136, 6, 14), (36, 264, 5, 10)])
@pytest.mark.parametrize("cc", [False, True])
@pytest.mark.parametrize("clip", [False, True])
def test_decisions(w, h, log2, bd, cc, clip):
    rec, fa = W.make_workload(7000 + w + bd, w, h, bd, log2, n_chroma_alt=5, ccalf=True)
    rng = np.random.default_rng(w)
    mx = (1 << bd) - 1
    src = rec.copy()
    for s, r in zip(src.planes(), rec.planes()):
        s[...] = np.clip(r.astype(np.int64) + rng.integers(-9, 10, size=r.shape), 0, mx)
    pre = np.ascontiguousarray(np.clip(rec.luma.astype(np.int64) + rng.integers(-5, 6, size=rec.luma.shape), 0, mx)
                               .astype(np.uint16))
    ctb = 1 << log2
    wc, hc = -(-w // ctb), -(-h // ctb)
    bounds = dict(clip_cols=[0] + [ctb] * (wc > 1) + [w], clip_rows=[0] + [ctb] * (hc > 1) + [h]) if clip else {}
    with native.Context(0) as ctx:
        for component in (1, 2):
            kw = dict(component=component, cc=cc, ctb_log2=log2, bit_depth=bd, pre_luma=pre if cc else None, **bounds)
            want, got = rec.copy(), rec.copy()
            dw, dg = (np.zeros(wc * hc, dtype=abi.ALF_CTB) for _ in range(2))
            oracle.chroma_alf_decide(src, want, dw, fa.apses[0], **kw)
            native.chroma_alf_decide(ctx, src, got, dg, fa.apses[0], **kw)
            assert dw.tobytes() == dg.tobytes()
            assert got.equal(want)
