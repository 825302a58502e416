"""The encoder's SAO statistics and the chroma merge decided from them: regions
that leave partial pairs, rows and slices, every depth, and pictures near the
ends of the sample range, where candidates clip and are summed from the samples
or the picture goes to the diagonal launches."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import abi, native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


def pair(seed, w, h, bd, log2, level=None):
    rec, _ = W.make_workload(seed, w, h, bd, log2)
    rng = np.random.default_rng(seed)
    mx = (1 << bd) - 1
    if level is not None:  # move part of the picture to an end of the range
        for p in rec.planes():
            n = int(p.shape[1] * level)
            p[:, :n // 2] = rng.integers(0, 6, size=(p.shape[0], n // 2))
            p[:, n // 2:n] = mx - rng.integers(0, 6, size=(p.shape[0], n - n // 2))
    src = rec.copy()
    for s, r in zip(src.planes(), rec.planes()):
        s[...] = np.clip(r.astype(np.int64) + rng.integers(-9, 10, size=r.shape), 0, mx)
    return src, rec


CASES = [(416, 240, 8, 7, None), (200, 136, 10, 5, None), (202, 138, 12, 6, None), (134, 70, 14, 6, None),
         (130, 66, 16, 7, None), (1030, 20, 10, 4, None), (416, 240, 10, 5, 0.04), (416, 240, 10, 6, 0.9),
         (256, 192, 8, 5, 0.05)]


@pytest.mark.parametrize("w,h,bd,log2,level", CASES)
def test_decision_and_merge(w, h, bd, log2, level):
    src, rec = pair(900 + w + bd, w, h, bd, log2, level)
    want = oracle.sao_decide_picture(src, rec, ctb_log2=log2, bit_depth=bd, params_dtype=abi.SAO_CTB_PARAMS)
    wc, hc = -(-w // (1 << log2)), -(-h // (1 << log2))
    with native.Context(0) as ctx:
        for device in (False, True):
            s, r = (native.DevicePicture.from_host(p) for p in (src, rec)) if device else (src, rec)
            got = native.sao_decide_picture(ctx, s, r, ctb_log2=log2, bit_depth=bd)
            assert got.tobytes() == np.ascontiguousarray(want).reshape(-1).tobytes()
            m, where = native.sao_chroma_merge(ctx, s, r, got, wc, hc, bit_depth=bd, ctb_log2=log2)
            om, owhere = oracle.sao_chroma_merge(src, rec, got, wc, hc, bit_depth=bd, ctb_log2=log2)
            assert np.array_equal(where, owhere) and m.tobytes() == om.tobytes()


def test_large_offsets_and_batch():
    """Offsets far above the decision's, and a batch whose second picture clips everywhere."""
    jobs = [pair(950, 256, 192, 10, 5), pair(951, 192, 128, 10, 5, 1.0), pair(952, 130, 130, 10, 5, 0.03)]
    rng = np.random.default_rng(3)
    with native.Context(0) as ctx:
        inds, grids = [], []
        for s, r in jobs:
            grid = (-(-s.width // 32), -(-s.height // 32))
            ind = np.array(W._sao_params(rng, grid[1], grid[0], 10)).reshape(-1)
            ind["cb"]["offset_val"] *= 9
            inds.append(np.ascontiguousarray(ind))
            grids.append(grid)
        devs = [(native.DevicePicture.from_host(s), native.DevicePicture.from_host(r)) for s, r in jobs]
        got = native.sao_chroma_merge_batch(ctx, [d[0] for d in devs], [d[1] for d in devs], inds, grids, bit_depth=10,
                                            ctb_log2=5)
    for (s, r), ind, grid, (m, where) in zip(jobs, inds, grids, got):
        om, owhere = oracle.sao_chroma_merge(s, r, ind, *grid, bit_depth=10, ctb_log2=5)
        assert np.array_equal(where, owhere) and m.tobytes() == om.tobytes()
