"""The server's parameter tables hold a full batch from the start, whatever the
requests' formats: a table that grows while requests are in flight synchronises
the device and allocates pinned memory."""
import numpy as np
import pytest

import oracle
from oxideav_h266_b200 import native
from oxideav_h266_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_sideinfo", [False, True])
def test_full_batch_allocates_nothing(device_sideinfo):
    import torch

    n = 2200
    big = W.make_workload(70, 3840, 2160, 10, 7)
    small, fa = W.make_workload(71, 32, 32, 10, 5)
    small, fa = W.with_chroma_format(small, fa, 3, 1)  # strips, luma tiles and full-height chroma tiles
    want = small.copy()
    oracle.apply_in_loop_filters(want, fa)
    with native.Context(0) as ctx:
        first = [(ctx.plan(*big), native.DevicePicture.from_host(big[0])) for _ in range(12)]
        rest = [(ctx.plan(small, fa, device_sideinfo=device_sideinfo), native.DevicePicture.from_host(small))
                for _ in range(n)]
        # a budget of one large request: they run one by one, and the others queue up behind them into one batch
        budget = 2 * sum(p.nbytes for p in big[0].planes())
        with native.Server(0, max_batch=n, memory_budget=budget) as srv:
            srv.set_batch_pixels(0)
            warm = first[:2] + rest[:n // 10]  # every kernel loaded, batched ones included
            srv.replay(*zip(*warm), np.zeros(len(warm)))
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            items = first + rest[n // 10:]
            srv.replay(*zip(*items), np.zeros(len(items)))
            torch.cuda.synchronize()
            assert torch.cuda.mem_get_info()[0] == free
        ctx.synchronize()
        assert all(d.to_host().equal(want) for _, d in rest[::99])
