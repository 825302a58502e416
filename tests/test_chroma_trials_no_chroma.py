"""The encoder's chroma ALF and CC-ALF decisions of CTBs without chroma samples:
odd luma sizes with halved chroma rounded down leave the last CTB column and row
without any, and they keep "off" whatever the work memory held before."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import abi, native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2", [5, 6, 7])
@pytest.mark.parametrize("cc", [False, True])
def test_last_ctbs_stay_off(log2, cc):
    ctb = 1 << log2
    w, h = 256 + 1, 128 + 1
    full, fa = W.make_workload(40 + log2, 264, 136, 10, log2, n_chroma_alt=5, ccalf=True)
    crop = lambda p: W.PictureData(*(np.ascontiguousarray(a[:n, :m]) for a, n, m in
                                     zip(p.planes(), (h, h // 2, h // 2), (w, w // 2, w // 2))), 10)
    rec = crop(full)
    rng = np.random.default_rng(log2)
    src = rec.copy()
    for s, r in zip(src.planes(), rec.planes()):
        s[...] = np.clip(r.astype(np.int64) + rng.integers(-9, 10, size=r.shape), 0, 1023)
    pre = rec.luma.copy()
    wc, hc = -(-w // ctb), -(-h // ctb)
    aps = fa.apses[0]
    with native.Context(0) as ctx:
        for component in (1, 2):
            kw = dict(component=component, cc=cc, ctb_log2=log2, bit_depth=10, pre_luma=pre if cc else None)
            # another call's results in the work memory: counts, seldom -1
            native.sao_decide_picture(ctx, full, full, ctb_log2=log2, bit_depth=10)
            want, got = rec.copy(), rec.copy()
            dw, dg = (np.zeros(wc * hc, dtype=abi.ALF_CTB) for _ in range(2))
            oracle.chroma_alf_decide(src, want, dw, aps, **kw)
            native.chroma_alf_decide(ctx, src, got, dg, aps, **kw)
            assert dw.tobytes() == dg.tobytes()
            assert got.equal(want)
