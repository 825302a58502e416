"""Batches that list a picture, or pictures with common samples, more than once with
deblocking in place among them: the items run as listed, as single executions do.
(Pictures that share nothing, views of one surface among them, stay in the
batched launches.)"""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


def make(cfi, seed=90):
    pic, fa = W.make_workload(seed, 264, 136, 10, 6, inter_frac=0.3, ccalf=True)
    if cfi != 1:
        pic, fa = W.with_chroma_format(pic, fa, cfi, 2)
    return pic, fa


def deblock_only(cfi):
    _, fa = make(cfi)
    fa.sao = fa.alf = fa.lmcs = None
    return fa


@pytest.mark.parametrize("cfi", [1, 3])
@pytest.mark.parametrize("device_sideinfo", [False, True])
def test_in_place_before_the_whole_chain(cfi, device_sideinfo):
    pic, full = make(cfi)
    want = pic.copy()
    oracle.apply_in_loop_filters(want, deblock_only(cfi))
    oracle.apply_in_loop_filters(want, full)
    other, other_fa = make(cfi, 91)
    other_want = other.copy()
    oracle.apply_in_loop_filters(other_want, other_fa)
    with native.Context(0) as ctx:
        plans = [ctx.plan(p, f, device_sideinfo=device_sideinfo)
                 for p, f in ((other, other_fa), (pic, deblock_only(cfi)), (pic, full))]
        for _ in range(20):
            dev, dev2 = native.DevicePicture.from_host(pic), native.DevicePicture.from_host(other)
            ctx.execute_plans(plans, [dev2, dev, dev])
            ctx.synchronize()
            assert dev.to_host().equal(want) and dev2.to_host().equal(other_want)


@pytest.mark.parametrize("device_sideinfo", [False, True])
def test_in_place_twice_with_common_chroma(device_sideinfo):
    """Two pictures of one luma plane each whose Cb is the same memory."""
    pic, fa = make(1)[0], deblock_only(1)
    want = pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    twice = W.PictureData(pic.luma.copy(), want.cb.copy(), want.cr.copy(), 10)
    oracle.apply_in_loop_filters(twice, fa)
    with native.Context(0) as ctx:
        plans = [ctx.plan(pic, fa, device_sideinfo=device_sideinfo) for _ in range(2)]
        for _ in range(20):
            a, b = native.DevicePicture.from_host(pic), native.DevicePicture.from_host(pic)
            b.cb = a.cb
            ctx.execute_plans(plans, [a, b])
            ctx.synchronize()
            got_a, got_b = a.to_host(), b.to_host()
            assert (got_a.luma == want.luma).all() and (got_a.cr == want.cr).all()
            assert (got_b.luma == want.luma).all() and (got_b.cr == want.cr).all()
            assert (got_a.cb == twice.cb).all()


class View(native.DevicePicture):
    """Planes that are views of larger ones: rows `stride(0)` samples apart."""

    def to_ctypes(self):
        pic = super().to_ctypes()
        for name in ("luma", "cb", "cr"):
            getattr(pic, name).stride = getattr(self, name).stride(0)
        return pic


def test_views_of_one_surface_share_launches():
    import torch

    pic, fa = make(1)[0], deblock_only(1)
    want = pic.copy()
    oracle.apply_in_loop_filters(want, fa)
    with native.Context(0) as ctx:
        plans = [ctx.plan(pic, fa) for _ in range(4)]
        devs = [native.DevicePicture.from_host(pic) for _ in range(4)]
        torch.cuda.synchronize()
        before = ctx.kernel_launches
        ctx.execute_plans(plans, devs)
        ctx.synchronize()
        apart = ctx.kernel_launches - before
        surface = [torch.from_numpy(p.view("int16")).cuda().repeat(2, 2) for p in pic.planes()]
        views = [View(*(s[y * p.shape[0]:(y + 1) * p.shape[0], x * p.shape[1]:(x + 1) * p.shape[1]]
                        for s, p in zip(surface, pic.planes())), 10) for y in (0, 1) for x in (0, 1)]
        torch.cuda.synchronize()
        before = ctx.kernel_launches
        ctx.execute_plans(plans, views)
        ctx.synchronize()
        assert ctx.kernel_launches - before == apart
    for s, p in zip(surface, want.planes()):
        assert (s.cpu().numpy().view("uint16") == np.tile(p, (2, 2))).all()
