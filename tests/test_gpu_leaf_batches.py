"""Batched triangle tests of the traversal kernel (k_trace): leaves wait in a ring
per warp and are tested 32 at a time, or fewer before a refill and when lanes are
idle.  Stacks of triangles make every ray reach many leaves at once, around the
sizes of a batch and of the ring; the records must be the oracle's, bit for bit."""
import numpy as np
import pytest

from rtcgb import rays as R

pytestmark = pytest.mark.gpu


def _stack(layers):
    """`layers` parallel triangles over the unit square, spaced in z, slightly turned."""
    rng = np.random.default_rng(layers)
    v = np.zeros((layers, 3, 3), np.float32)
    v[:, 0] = (-1.0, -1.0, 0.0)
    v[:, 1] = (3.0, -1.0, 0.0)
    v[:, 2] = (-1.0, 3.0, 0.0)
    v += rng.uniform(-0.05, 0.05, v.shape).astype(np.float32)
    v[:, :, 2] += (np.arange(layers, dtype=np.float32) * 0.25)[:, None]
    return v.reshape(-1, 3), np.arange(3 * layers, dtype=np.uint32).reshape(-1, 3)


def _rays(n, layers, seed):
    """Rays through the stack from below, from above and sideways; a few end before the first layer."""
    rng = np.random.default_rng(seed)
    top = layers * 0.25 + 1.0
    org = rng.uniform(0.0, 1.0, (n, 3))
    org[:, 2] = np.where(rng.random(n) < 0.5, -1.0, top)
    d = rng.uniform(-0.3, 0.3, (n, 3))
    d[:, 2] = np.where(org[:, 2] < 0, 1.0, -1.0)
    d[rng.random(n) < 0.1, 2] *= 0.01
    r = R.make_rayhits(org, d)
    r["tfar"][rng.random(n) < 0.2] = 0.4
    return r


@pytest.mark.parametrize("robust", [False, True])
@pytest.mark.parametrize("leaf_max", [1, 4])
@pytest.mark.parametrize("layers", [1, 9, 31, 32, 33, 65, 300])
def test_stacked_leaves_match_oracle(rtc, oracle, layers, leaf_max, robust):
    dev = rtc.Device(f"gpu.leaf_max={leaf_max}".encode())
    verts, idx = _stack(layers)
    sc = rtc.Scene(dev, flags=rtc.RTC_SCENE_FLAG_ROBUST if robust else 0)
    sc.add_mesh(verts, idx)
    sc.commit()
    orc = oracle.OracleScene([(0, verts, idx)], robust=robust)
    for n in (1, 31, 33, 1000):
        rays = _rays(n, layers, seed=n)
        got, ref = rays.copy(), rays.copy()
        sc.intersect(got)
        orc.intersect(ref)
        assert R.hits_equal_bits(got, ref).all()
        shadow = R.make_rays(np.stack([rays["org_x"], rays["org_y"], rays["org_z"]], -1),
                             np.stack([rays["dir_x"], rays["dir_y"], rays["dir_z"]], -1), 0.0, rays["tfar"])
        got, ref = shadow.copy(), shadow.copy()
        sc.occluded(got)
        orc.occluded(ref)
        assert np.array_equal(got["tfar"], ref["tfar"])
    sc.release()
    dev.release()
