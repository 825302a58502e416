"""Which deblocking segments depend on each other, and the tile kernel's two
regions.

A luma segment of maxFilterLength m on a side writes m samples there and uses
m + 1 (three at least), chroma writes 3 and uses 4
(src/deblock.rs:1224-1776, 1803-2075).  Segments of a pass between which nobody
writes what another uses commute: the oracle's own segment log, replayed in a
shuffled order, must reproduce its output.  Pictures whose segments are all
independent (h266_sideinfo_mode 1) are checked segment by segment, the others
component by component."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import abi, native
from oxideav_h266_b200 import workloads as W

TILES, STRIPS = 1, 2


def spans(r):
    """(write start, write end, use start, use end) along the edge normal of a log row."""
    pos = int(r[2] if r[1] else r[3])
    mp, mq = int(r[5]), int(r[6])

    def w(m, other):
        return 3 if r[0] else max(max(m, 3) if other > 3 else m, 1)

    wp, wq = w(mp, mq), w(mq, mp)
    rp, rq = (3 if x <= 2 else x + 1 for x in (wp, wq))
    return pos - wp, pos + wq, pos - rp, pos + rq


def filtering(log):
    return [i for i, r in enumerate(log) if r[8] != 0 and not (r[0] != 0 and r[5] == 1 and r[6] == 1 and r[4] != 2)]


def components(log):
    """Per pass, the components of every band (emission order inside)."""
    out = {0: [], 1: []}
    bands = {}
    for i in filtering(log):
        r = log[i]
        bands.setdefault((int(r[1]), int(r[0]), int(r[3] if r[1] else r[2])), []).append(i)
    for (vert, _, _), idx in bands.items():
        idx.sort(key=lambda i: (int(log[i][2] if vert else log[i][3]), i))
        sp = [spans(log[i]) for i in idx]
        cur = [idx[0]]
        for k in range(1, len(idx)):
            cut = max(s[1] for s in sp[:k]) <= min(s[2] for s in sp[k:]) and \
                max(s[3] for s in sp[:k]) <= min(s[0] for s in sp[k:])
            if cut:
                out[0 if vert else 1].append(sorted(cur))
                cur = []
            cur.append(idx[k])
        out[0 if vert else 1].append(sorted(cur))
    return out


def replay(pic, fa, comps, log, seed):
    rng = np.random.default_rng(seed)
    order = [i for p in (0, 1) for ci in rng.permutation(len(comps[p])) for i in comps[p][ci]]
    got = pic.copy()
    oracle.deblock_replay(got, log, np.array(order, dtype=np.uint64))
    return got


def on_sub_block_grid(fa):
    """Drops the TB splits that put a transform edge beside the sub-block grid of their CU."""
    cus = fa.cus
    for i in np.nonzero((cus["has_num_sb"] != 0) & (cus["has_tb_split"] != 0))[0]:
        dim = int(cus["w"][i] if cus["ts_vertical"][i] else cus["h"][i])
        nsb = max(int(cus["num_sb_x"][i] if cus["ts_vertical"][i] else cus["num_sb_y"][i]), 1)
        sb, last = max(8, dim // nsb), min(max(dim // 8, 1) - 1, nsb - 1)
        b = cus["ts_bounds"][i][: cus["ts_n_bounds"][i]]
        if last and any(int(x) % sb or int(x) // sb > last for x in b):
            cus["has_tb_split"][i] = 0
    return fa


def narrow(seed, w, h, **kw):
    """Multi-type-tree picture with 4-sample CUs, TB splits and sub-block grids whose segments are independent."""
    pic, fa = W.stress_workload(seed, w, h, **kw)
    cus = fa.cus
    for i in np.nonzero((cus["has_num_sb"] != 0) & (cus["has_tu64"] != 0))[0]:
        cus["has_tu64"][i] = 0
    return pic, on_sub_block_grid(fa)


def all_4x4(seed, w, h):
    """Every CU 4x4: the most segments a tile can have on the 4x4 grid."""
    pic, fa = W.make_workload(seed, w, h, 10, 5, ccalf=True, lmcs=True)
    ys, xs = np.mgrid[0:h:4, 0:w:4]
    cus = np.zeros(xs.size, dtype=abi.DEBLOCK_CU)
    cus["x"], cus["y"], cus["w"], cus["h"] = xs.reshape(-1), ys.reshape(-1), 4, 4
    cus["qp_y"] = 37
    cus["qp_c"][:, :] = abi.DEBLOCK_QP_C_LEGACY
    cus["intra"] = 1
    fa.cus, fa.mv = cus, None
    return pic, fa


def all_8x8(seed, w, h):
    """Every CU 8x8: the most segments a tile can have on the 8x8 grid."""
    pic, fa = W.make_workload(seed, w, h, 10, 6, ccalf=True, lmcs=True)
    ys, xs = np.mgrid[0:h:8, 0:w:8]
    cus = np.zeros(xs.size, dtype=abi.DEBLOCK_CU)
    cus["x"], cus["y"], cus["w"], cus["h"] = xs.reshape(-1), ys.reshape(-1), 8, 8
    cus["qp_y"] = 37
    cus["qp_c"][:, :] = abi.DEBLOCK_QP_C_LEGACY
    cus["intra"] = 1
    fa.cus, fa.mv = cus, None
    return pic, fa


def wide_between(seed, w, h):
    """32-sample CUs 4 samples off the tile grid beside 4-sample ones: long filters that reach across tile borders."""
    pic, fa = W.make_workload(seed, w, h, 10, 6, ccalf=True, lmcs=True)
    xs = [0] + list(range(4, w - 32, 32))
    ys = [0] + list(range(4, h - 32, 32))
    xw = [4] + [32] * (len(xs) - 2) + [w - xs[-1]]
    yh = [4] + [32] * (len(ys) - 2) + [h - ys[-1]]
    cus = np.zeros(len(xs) * len(ys), dtype=abi.DEBLOCK_CU)
    cus["x"], cus["w"] = np.tile(xs, len(ys)), np.tile(xw, len(ys))
    cus["y"], cus["h"] = np.repeat(ys, len(xs)), np.repeat(yh, len(xs))
    cus["qp_y"] = 40
    cus["qp_c"][:, :] = abi.DEBLOCK_QP_C_LEGACY
    cus["intra"] = 1
    fa.cus, fa.mv = cus, None
    return pic, fa


@pytest.mark.parametrize("seed", range(12))
def test_independent_segments_replay_in_any_order(seed):
    pic, fa = narrow(seed, 192, 128, bit_depth=8 + 2 * (seed % 2), dual_tree=seed % 3 == 1)
    assert native.sideinfo_mode(pic, fa) == TILES
    want = pic.copy()
    oracle.apply_deblocking_clipped(want, fa)
    log = oracle.deblock_edge_log(pic, fa)
    comps = components(log)
    assert max(len(c) for c in comps[0] + comps[1]) == 1
    assert replay(pic, fa, comps, log, seed).equal(want)


@pytest.mark.parametrize("seed", range(8))
def test_components_by_spans_replay_in_any_order(seed):
    pic, fa = W.stress_workload(500 + seed, 192, 128)
    want = pic.copy()
    oracle.apply_deblocking_clipped(want, fa)
    log = oracle.deblock_edge_log(pic, fa)
    comps = components(log)
    if native.sideinfo_mode(pic, fa) == TILES:  # never where segments depend on each other
        assert max(len(c) for c in comps[0] + comps[1]) == 1
    assert replay(pic, fa, comps, log, seed).equal(want)


PICTURES = {
    "narrow_192x128": lambda: narrow(40, 192, 128),
    "narrow_200x136": lambda: narrow(41, 200, 136, ctb_log2=5),
    "narrow_132x68": lambda: narrow(42, 132, 68, ctb_log2=5),
    "narrow_dual_8bit": lambda: narrow(43, 256, 192, dual_tree=True, bit_depth=8),
    "narrow_tiles": lambda: narrow(44, 256, 192, tiles=True, ctb_log2=5),
    "all_4x4_136": lambda: all_4x4(45, 136, 136),
    "all_8x8_136": lambda: all_8x8(46, 136, 136),
    "wide_200": lambda: wide_between(47, 200, 200),
    "wide_64": lambda: wide_between(48, 64, 72),
    "chains": lambda: W.stress_workload(3000, 1100, 100),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(PICTURES))
def test_gpu_regions_and_runs(name):
    """The chain with device-built and host-built side information, alone and in a batch, against the oracle."""
    pic, fa = PICTURES[name]()
    want = pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    assert native.sideinfo_mode(pic, fa) == (STRIPS if name == "chains" else TILES)
    with native.Context(0) as ctx:
        got = pic.copy()
        ctx.apply_in_loop_filters(got, fa)
        assert got.equal(want), "device-built, one picture"
        for device in (False, True):
            plans = [ctx.plan(pic, fa, device_sideinfo=device) for _ in range(2)]
            devs = [native.DevicePicture.from_host(pic) for _ in plans]
            ctx.execute_plans(plans, devs)
            ctx.synchronize()
            assert all(d.to_host().equal(want) for d in devs), f"batch, device-built {device}"
