"""The plain form of the clipped ALF taps, which tiles with samples of 2^14 or above
take: differences of neighbours up to 65535, in luma and in the chroma of every
format."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bd", [8, 10, 14])
@pytest.mark.parametrize("cfi", [1, 2, 3])
@pytest.mark.parametrize("value", [20000, 32768, 40000, 65535])
def test_far_neighbours(bd, cfi, value):
    pic, fa = W.make_workload(20 + bd, 200, 136, bd, 6, ccalf=True, n_luma_aps=2, n_chroma_alt=2, alf_fixed_frac=0.3)
    if cfi != 1:
        pic, fa = W.with_chroma_format(pic, fa, cfi, 3)
    fa.deblock.disabled = 1
    fa.sao[:] = np.zeros_like(fa.sao)
    rng = np.random.default_rng(value)
    for p in pic.planes():
        y, x = np.mgrid[0:p.shape[0], 0:p.shape[1]]
        flip = rng.random(p.shape) < 0.3
        p[...] = np.where(x < p.shape[1] // 2, np.where(((x + y) & 1).astype(bool) ^ flip, value, p), p)
    want, got = pic.copy(), pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    with native.Context(0) as ctx:
        ctx.apply_in_loop_filters(got, fa)
    assert got.equal(want)
