"""The strip kernels from several threads at once: planes of different heights
need different amounts of shared memory, and no launch depends on what another
thread's launch asked for."""
import ctypes as C
import threading

import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_sideinfo", [False, True])
def test_heights_side_by_side(device_sideinfo):
    failed, done = [], []

    def work(h):
        pic, fa = W.make_workload(h, 64, h, 10, 6)
        fa.sao = fa.alf = None  # deblocked in place, by the strips
        want = pic.copy()
        oracle.apply_in_loop_filters(want, fa)
        try:
            with native.Context(0) as ctx:
                plan, dev = ctx.plan(pic, fa, device_sideinfo=device_sideinfo), native.DevicePicture.from_host(pic)
                cp = C.byref(dev.to_ctypes())
                ready.wait()
                for _ in range(100):
                    for _ in range(40):
                        if native.lib().h266_chain_plan_execute(ctx._h, plan._h, cp):
                            raise native.H266Error(0, native.lib().h266_last_error().decode())
                    ctx.synchronize()
                last = native.DevicePicture.from_host(pic)
                plan.execute(last)
                ctx.synchronize()
                done.append(last.to_host().equal(want))
        except native.H266Error as e:
            failed.append(str(e))

    heights = (4096, 3200, 2304)
    ready = threading.Barrier(len(heights), timeout=60)
    threads = [threading.Thread(target=work, args=(h,)) for h in heights]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    assert done == [True] * len(heights)
