"""A captured build replayed on input with another number of valid triangles than it was
captured for, falling and growing: the replay must not be taken for a build (its
arrays are sized for the planned count), the commit builds the ordinary way, and the
hits are the oracle's.  On both sides of the size that one CTA clusters alone."""
import numpy as np
import pytest

from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu


def _check(sc, oracle, meshes, seed):
    rays = W.sphere_rays(3000, seed=seed)
    got, ref = rays.copy(), rays.copy()
    sc.intersect(got)
    oracle.OracleScene(meshes).intersect(ref)
    assert R.hits_equal_bits(got, ref).all()


@pytest.mark.parametrize("config", [b"", b"gpu.ploc_radius=4", b"gpu.collapse=greedy"])
@pytest.mark.parametrize("tris", [200, 4096, 5000, 40_000])
@pytest.mark.parametrize("gone", [1, 100, -1])
def test_commits_with_fewer_then_more_valid_triangles(rtc, oracle, config, tris, gone):
    gone = gone if gone > 0 else tris - 1  # all but one
    v, i = W.gaussian_soup(tris, seed=tris)
    bad = v.copy()
    bad[: 3 * gone] = np.nan
    dev = rtc.Device(config)
    sc = rtc.Scene(dev)
    sc.add_mesh(v.copy(), i)
    # valid until captured; fewer (captured anew); as many; all valid again; fewer
    for k, verts in enumerate([v, v, v, bad, bad, v, v, v, bad, v]):
        sc.update_vertices(0, verts)
        sc.commit()
        assert sc.build_stats()["num_prims"] == (tris if verts is v else tris - gone)
        _check(sc, oracle, [(0, verts, i)], k)
    sc.release()
    dev.release()


def test_batched_frame_whose_count_grows(rtc):
    """A frame captured with some triangles invalid, replayed with them valid (written to
    the device buffers in place), reports the mismatch and traces nothing; with the
    planned count again it gives the first frame's bytes."""
    torch = pytest.importorskip("torch")
    dev = rtc.Device(b"")
    meshes = [W.gaussian_soup(n, seed=n) for n in (6000, 300, 20_000)]
    sc = rtc.Scene(dev)
    sc.set_batched()
    whole, bufs = [], []
    for v, i in meshes:
        t = torch.from_numpy(v.copy()).cuda()
        whole.append(t.clone())
        t[: 3 * 150] = float("nan")
        idx = torch.from_numpy(i.astype(np.int32)).cuda()
        torch.cuda.synchronize()
        bufs.append((t, idx))
        sc.add_mesh_device(t.data_ptr(), t.shape[0], idx.data_ptr(), idx.shape[0])
    sc.commit()
    rays = W.sphere_rays(9000, seed=3)
    start = np.array([0, 3000, 6000, 9000], np.uint32)
    fresh = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    work = torch.zeros_like(fresh)
    frame = rtc.BatchedFrame(sc, work.data_ptr(), 9000, start, pristine_ptr=fresh.data_ptr())
    frame.replay()
    first = work.cpu().numpy().copy()
    assert (first.reshape(-1).view(R.RAYHIT_DTYPE)["geomID"] != R.RTC_INVALID_GEOMETRY_ID).any()
    for (t, _), w in zip(bufs, whole):
        t.copy_(w)
    torch.cuda.synchronize()
    with pytest.raises(rtc.RTCError):
        frame.replay()
    assert np.array_equal(work.cpu().numpy(), rays.view(np.uint8))
    for t, _ in bufs:
        t[: 3 * 150] = float("nan")
    torch.cuda.synchronize()
    frame.replay()
    assert np.array_equal(work.cpu().numpy(), first)
    frame.release()
    sc.release()
    dev.release()
