"""The chroma SAO merge at its limits: more CTB rows than the wavefront takes
(anti-diagonal launches alone, without the statistics and their memory) and a
batch of more pictures than one launch dimension holds."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


def job(seed, w, h, log2):
    rec, _ = W.make_workload(seed, w, h, 10, 5)
    rng = np.random.default_rng(seed)
    src = rec.copy()
    for s, r in zip(src.planes(), rec.planes()):
        s[...] = np.clip(r.astype(np.int64) + rng.integers(-9, 10, size=r.shape), 0, 1023)
    grid = (-(-w // (1 << log2)), -(-h // (1 << log2)))
    return src, rec, np.ascontiguousarray(np.array(W._sao_params(rng, grid[1], grid[0], 10)).reshape(-1)), grid


@pytest.mark.parametrize("h,diagonals", [(1024, False), (1028, True)])
def test_many_ctb_rows(h, diagonals):
    src, rec, ind, grid = job(980, 64, h, 2)
    want, where = oracle.sao_chroma_merge(src, rec, ind, *grid, bit_depth=10, ctb_log2=2)
    with native.Context(0) as ctx:
        s, r = native.DevicePicture.from_host(src), native.DevicePicture.from_host(rec)
        before = ctx.kernel_launches
        got, gwhere = native.sao_chroma_merge(ctx, s, r, ind, *grid, bit_depth=10, ctb_log2=2)
        launches = ctx.kernel_launches - before
    assert np.array_equal(gwhere, where) and got.tobytes() == want.tobytes()
    assert launches == (grid[0] + grid[1] - 1 if diagonals else 2)


def test_large_batch():
    src, rec, ind, grid = job(981, 16, 8, 5)
    want, where = oracle.sao_chroma_merge(src, rec, ind, *grid, bit_depth=10, ctb_log2=5)
    n = 65537
    with native.Context(0) as ctx:
        s, r = native.DevicePicture.from_host(src), native.DevicePicture.from_host(rec)
        out = native.sao_chroma_merge_batch(ctx, [s] * n, [r] * n, [ind] * n, [grid] * n, bit_depth=10, ctb_log2=5)
    assert all(np.array_equal(m, where) and g.tobytes() == want.tobytes() for g, m in out)
