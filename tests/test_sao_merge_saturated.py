"""The chroma SAO merge where a CTB's component holds nothing but the largest
(or smallest) sample: such CTBs have samples like any other, and the parameters
they could take over change their error."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import abi, native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


def merged_as_oracle(src, rec, ind, grid, bd, log2):
    want, where = oracle.sao_chroma_merge(src, rec, ind, *grid, bit_depth=bd, ctb_log2=log2)
    with native.Context(0) as ctx:
        got, gwhere = native.sao_chroma_merge(ctx, src, rec, ind, *grid, bit_depth=bd, ctb_log2=log2)
        s, r = native.DevicePicture.from_host(src), native.DevicePicture.from_host(rec)
        [(b, bwhere)] = native.sao_chroma_merge_batch(ctx, [s], [r], [ind], [grid], bit_depth=bd, ctb_log2=log2)
    assert np.array_equal(gwhere, where) and got.tobytes() == want.tobytes()
    assert np.array_equal(bwhere, where) and b.tobytes() == want.tobytes()
    return where


@pytest.mark.parametrize("bd", [10, 14, 15, 16])
def test_flat_white_keeps_its_own(bd):
    """A band offset of -35 over the only band would cost more than a CTB's own parameters."""
    mx = (1 << bd) - 1
    pic = W.PictureData(*(np.full(s, mx, dtype=np.uint16) for s in ((32, 64), (16, 32), (16, 32))), bd)
    ind = np.zeros(2, dtype=abi.SAO_CTB_PARAMS)
    ind["cb"]["sao_type_idx"][0], ind["cb"]["band_position"][0], ind["cb"]["offset_val"][0] = 1, 31, [0, -35, 0, 0, 0]
    assert list(merged_as_oracle(pic, pic.copy(), ind, (2, 1), bd, 5)) == [0, 0]


@pytest.mark.parametrize("bd", [8, 14, 16])
@pytest.mark.parametrize("planes", [(1,), (2,), (1, 2)])
@pytest.mark.parametrize("level", ["top", "bottom"])
def test_flat_ctbs_among_others(bd, planes, level):
    w, h, log2 = 200, 136, 5
    mx = (1 << bd) - 1
    rec, _ = W.make_workload(970 + bd, w, h, bd, log2)
    rng = np.random.default_rng(bd + len(planes))
    grid = (-(-w // 32), -(-h // 32))
    src = rec.copy()
    for k, (s, r) in enumerate(zip(src.planes(), rec.planes())):
        if k in planes:
            for _ in range(9):  # whole CTBs of one sample value, the original a little inside the range
                x, y = 16 * int(rng.integers(grid[0])), 16 * int(rng.integers(grid[1]))
                r[y:y + 16, x:x + 16] = mx if level == "top" else 0
        s[...] = np.clip(r.astype(np.int64) + rng.integers(-9, 10, size=r.shape), 0, mx)
    ind = np.ascontiguousarray(np.array(W._sao_params(rng, grid[1], grid[0], bd)).reshape(-1))
    merged_as_oracle(src, rec, ind, grid, bd, log2)
