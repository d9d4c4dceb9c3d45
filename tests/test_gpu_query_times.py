"""Times in the query statistics: total_ms covers everything that a call enqueues -- the
set-up of a thread's first query, the batch boundaries, the rays' copies -- and
kernel_ms the traversal alone."""
import threading

import numpy as np
import pytest

from rtcgb import workloads as W

pytestmark = pytest.mark.gpu


def test_total_covers_the_whole_call(rtc):
    import torch
    dev = rtc.Device(b"gpu.host_rays=copy")
    plain, batched = rtc.Scene(dev), rtc.Scene(dev)
    batched.set_batched()
    for sc in (plain, batched):
        sc.add_mesh(*W.gaussian_soup(3000, seed=5))
        sc.add_mesh(*W.heightfield(16))
        sc.commit()
    n = 5000
    rays = W.sphere_rays(n, seed=3)
    buf = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    seen = {}

    def calls():  # of a new thread: its scratch is not yet zero
        for k, call in enumerate([lambda: plain.intersect_ptr(buf.data_ptr(), n),
                                  lambda: plain.intersect_ptr(buf.data_ptr(), n),
                                  lambda: batched.intersect_batched(None, [0, 2000, n], ptr=buf.data_ptr(), count=n),
                                  lambda: plain.intersect(rays.copy())]):
            call()
            seen[k] = rtc.last_query_stats()

    t = threading.Thread(target=calls)
    t.start()
    t.join()
    assert sorted(seen) == [0, 1, 2, 3]
    assert all(s["total_ms"] >= s["kernel_ms"] > 0 for s in seen.values()), seen
    for k in (0, 2, 3):
        assert seen[k]["total_ms"] > seen[k]["kernel_ms"], seen[k]
    for sc in (plain, batched):
        sc.release()
    dev.release()
