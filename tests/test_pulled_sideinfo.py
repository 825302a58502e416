"""Side information that a kernel copies from pinned staging: groups of one
picture up to the full sixteen, sections of every remainder by 16 bytes, and
staging reused by a second, different batch."""
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


def make(seed):
    w, h = 64 + 8 * (seed % 5), 40 + 4 * (seed % 7)
    return W.make_workload(900 + seed, w, h, 8 + 2 * (seed % 2), 5 + seed % 2, inter_frac=0.3, ccalf=seed % 3 == 0,
                           lmcs=seed % 4 == 1)


@pytest.mark.parametrize("group,n", [(1, 3), (4, 17), (16, 16), (16, 33)])
def test_groups(group, n):
    with native.Context(0) as ctx:
        ctx.set_tuning("e2e_group", group)
        for base in (0, 50):
            items = [make(base + i) for i in range(n)]
            got = [p.copy() for p, _ in items]
            ctx.apply_in_loop_filters_batch(got, [f for _, f in items])
            for g, (p, f) in zip(got, items):
                want = p.copy()
                oracle.apply_in_loop_filters(want, f)
                assert g.equal(want)
