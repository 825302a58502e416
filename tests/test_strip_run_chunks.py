"""Runs of chained cells in the strip kernels where a band has more cells than
one staged chunk holds (640): wide pictures for the rows, tall ones for the
columns, sizes around the chunk's end."""
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(2552, 64), (2560, 40), (2568, 48), (2696, 64), (5200, 24), (64, 1280), (40, 1288),
                                 (24, 2700)])
def test_runs_across_chunks(w, h):
    pic, fa = W.stress_workload(w + h, w, h)
    assert native.sideinfo_mode(pic, fa) == 2
    want = pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    with native.Context(0) as ctx:
        got = pic.copy()
        ctx.apply_in_loop_filters(got, fa)
    assert got.equal(want)
