"""State that outlives a call: the per-thread query scratch that a kernel leaves zero
for the next launch, across all kinds of queries in any order; and the BVH of a
replayed rebuild, which stays in the captured build's arrays until the next one."""
import threading

import numpy as np
import pytest

from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu


def _mesh(n, seed):
    return W.gaussian_soup(n, seed=seed)


def _check(sc, orc, n, seed, how):
    import torch
    rays = W.sphere_rays(n, seed=seed)
    ref = rays.copy()
    orc.intersect(ref)
    if how == "device":
        buf = torch.from_numpy(rays.view(np.uint8).reshape(n, 80).copy()).cuda()
        torch.cuda.synchronize()
        sc.intersect_ptr(buf.data_ptr(), n)
        got = buf.cpu().numpy().reshape(-1).view(R.RAYHIT_DTYPE)
    elif how == "filter":
        got = rays.copy()
        sc.intersect(got, context_filter=lambda *a: True)
    else:
        got = rays.copy()
        sc.intersect(got)
    assert R.hits_equal_bits(got, ref).all(), how


@pytest.mark.parametrize("mode", [b"gpu.host_rays=direct", b"gpu.host_rays=copy", b"gpu.host_rays=pipeline"])
def test_queries_of_all_kinds_in_turn(rtc, oracle, mode):
    dev = rtc.Device(mode)
    verts, idx = _mesh(3000, 5)
    orc = oracle.OracleScene([(0, verts, idx)])
    plain = rtc.Scene(dev)
    plain.add_mesh(verts, idx)
    plain.commit()
    filtered = rtc.Scene(dev, flags=rtc.RTC_SCENE_FLAG_CONTEXT_FILTER_FUNCTION)
    filtered.add_mesh(verts, idx)
    filtered.commit()
    for k, (sc, n, how) in enumerate([(plain, 1, "device"), (plain, 500, "host"), (plain, 33, "device"),
                                      (filtered, 50, "filter"), (plain, 4000, "device"), (plain, 1, "host"),
                                      (plain, 2, "device")]):
        _check(sc, orc, n, 20 + k, how)
    failures = []

    def other():  # a new thread has a scratch of its own
        try:
            _check(plain, orc, 700, 99, "host")
            _check(plain, orc, 700, 98, "device")
        except BaseException as e:  # noqa: BLE001
            failures.append(e)

    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert not failures
    for sc in (plain, filtered):
        sc.release()
    dev.release()


def test_replayed_rebuilds_share_their_arrays(rtc, device, oracle):
    verts, idx = _mesh(20_000, 7)
    sc = rtc.Scene(device)
    gid = sc.add_mesh(verts, idx)
    for frame in range(5):
        moved = W.displace_soup(verts, 7 * frame)
        sc.update_vertices(gid, moved)
        sc.commit()
        _check(sc, oracle.OracleScene([(gid, moved, idx)]), 500, frame, "host")
    # another layout: the captured build goes, a new one is made after two commits
    more = _mesh(9_000, 8)
    g2 = sc.add_mesh(*more)
    for _ in range(4):
        sc.commit()
        _check(sc, oracle.OracleScene([(gid, moved, idx), (g2, *more)]), 500, 60, "host")
    nodes, tris = sc.bvh()
    assert tris.shape[0] == 29_000 and nodes.shape[0] == sc.build_stats()["num_nodes"]
    sc.release()
