"""Refit in one cooperative launch (k_refit_all): trees of one node, of narrow levels
only, of levels wider than the narrow limit, and of more levels than the launch
holds (refitted level by level); after moving the vertices the hits must be those
of the oracle built from the moved mesh, bit for bit."""
import numpy as np
import pytest

from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu


def _spread(n):
    return W.gaussian_soup(n, seed=n)


def _nested(n):
    """Triangles of geometrically growing size around one point: a deep, narrow tree."""
    rng = np.random.default_rng(n)
    size = np.exp(np.linspace(-8.0, 0.0, n))[:, None, None]
    v = rng.uniform(-1.0, 1.0, (n, 3, 3)) * size
    return v.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("mesh", [_spread, _nested], ids=["spread", "nested"])
@pytest.mark.parametrize("n", [1, 2, 33, 600, 20_000])
@pytest.mark.parametrize("robust", [False, True])
def test_refit_matches_oracle(rtc, device, oracle, mesh, n, robust):
    verts, idx = mesh(n)
    sc = rtc.Scene(device, flags=rtc.RTC_SCENE_FLAG_ROBUST if robust else 0)
    gid = sc.add_mesh(verts, idx, quality=rtc.RTC_BUILD_QUALITY_REFIT)
    sc.commit()
    for frame in (1, 2):
        moved = W.displace_soup(verts, 15 * frame, amplitude=0.003)
        sc.update_vertices(gid, moved)
        sc.commit()
        st = sc.build_stats()
        assert st["refit"] == 1
        orc = oracle.OracleScene([(0, moved, idx)], robust=robust)
        rays = W.sphere_rays(2000, seed=n + frame)
        if mesh is _nested:
            for f in ("org_x", "org_y", "org_z"):
                rays[f] = rays[f] * 2 - 1
        got, ref = rays.copy(), rays.copy()
        sc.intersect(got)
        orc.intersect(ref)
        assert R.hits_equal_bits(got, ref).all()
        # every triangle is inside the scene box that the refit reports
        lo, hi = sc.bounds()
        assert np.all(moved.min(0) >= lo) and np.all(moved.max(0) <= hi)
    sc.release()


def test_refit_of_a_tree_deeper_than_the_launch_holds(rtc, device, oracle):
    """Thousands of equal triangles collapse into a chain of levels."""
    n = 3000
    verts = np.tile(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), (n, 1))
    idx = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    sc = rtc.Scene(device)
    gid = sc.add_mesh(verts, idx, quality=rtc.RTC_BUILD_QUALITY_REFIT)
    sc.commit()
    depth = sc.build_stats()["depth"]
    moved = verts + np.repeat(np.linspace(0.0, 1.0, n, dtype=np.float32), 3)[:, None] * np.array([0, 0, 1], np.float32)
    sc.update_vertices(gid, moved)
    sc.commit()
    assert sc.build_stats()["refit"] == 1 and depth > 64
    orc = oracle.OracleScene([(0, moved, idx)])
    rng = np.random.default_rng(5)
    org = rng.uniform(0.0, 0.5, (500, 3)) - np.array([0, 0, 1.0])
    rays = R.make_rayhits(org, np.tile([0.0, 0.0, 1.0], (500, 1)))
    got, ref = rays.copy(), rays.copy()
    sc.intersect(got)
    orc.intersect(ref)
    assert R.hits_equal_bits(got, ref).all()
    sc.release()
