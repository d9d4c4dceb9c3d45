"""A warp waits for more idle lanes where its last rays were short.  When it fetches
rays must not show in the results: rays that miss the scene's box, rays that end after
a few nodes and rays that cross the whole soup, alone, in blocks of one kind and
interleaved, give each ray the same answer in every order."""
import numpy as np
import pytest

from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu


def _rays(n):
    rng = np.random.default_rng(n)
    kind = np.arange(n) * 3 // n  # blocks: misses, short, long
    org = rng.uniform(-1, 1, (n, 3))
    dirs = rng.normal(size=(n, 3))
    org[kind == 0] += 1000.0
    return org, dirs, np.where(kind == 1, 1e-3, np.inf)


@pytest.mark.parametrize("robust", [False, True])
@pytest.mark.parametrize("n", [1, 33, 4099, 60_000])
def test_order_of_rays(rtc, n, robust):
    dev = rtc.Device(b"")
    sc = rtc.Scene(dev, flags=rtc.RTC_SCENE_FLAG_ROBUST if robust else 0)
    sc.add_mesh(*W.gaussian_soup(30_000, seed=2))
    sc.commit()
    org, dirs, tfar = _rays(n)
    perm = np.random.default_rng(1).permutation(n)
    for make, query in ((R.make_rayhits, sc.intersect), (R.make_rays, sc.occluded)):
        blocks = make(org, dirs)
        blocks["tfar"] = tfar
        mixed = blocks[perm].copy()
        query(blocks)
        query(mixed)
        assert mixed.tobytes() == blocks[perm].tobytes()
    sc.release()
    dev.release()
