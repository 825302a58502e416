"""SAO of samples far outside the depth, as far apart as 16 bits hold: a 0 with
neighbours of 32767 is a valley like any other, and offsets onto large samples
clip, in the packed tiles of every chroma format."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bd", [8, 12])
@pytest.mark.parametrize("cfi", [1, 2, 3])
@pytest.mark.parametrize("values", [(32767,), (16384, 32768, 65535)])
@pytest.mark.parametrize("eo_class", [0, 1, 2, 3, None])
def test_far_samples(bd, cfi, values, eo_class):
    pic, fa = W.make_workload(30 + bd, 200, 136, bd, 6, n_luma_aps=1)
    if cfi != 1:
        pic, fa = W.with_chroma_format(pic, fa, cfi, 3)
    rng = np.random.default_rng(7)
    for p in pic.planes():
        p[:, 70:] = 0
        p[rng.integers(0, p.shape[0], 200), rng.integers(0, p.shape[1], 200)] = rng.choice(values, 200)
    if eo_class is not None:  # else the workload's own mix of types, copies among them
        for c in ("luma", "cb", "cr"):
            fa.sao[c]["sao_type_idx"] = 2
            fa.sao[c]["eo_class"] = eo_class
            fa.sao[c]["offset_val"] = [0, 2, 5, -3, -1]
    want, got = pic.copy(), pic.copy()
    oracle.apply_sao_clipped(want, fa)
    with native.Context(0) as ctx:
        ctx.apply_sao_clipped(got, fa)
        assert got.equal(want)
        got, want = pic.copy(), pic.copy()
        fa.alf_cfg.alf_enabled = 0
        fa.deblock.disabled = 1
        oracle.apply_in_loop_filters(want, fa)
        ctx.apply_in_loop_filters(got, fa)
        assert got.equal(want)
