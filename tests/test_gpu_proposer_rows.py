"""Proposer inference is row by row: a ray's proposals depend neither on how many rays
are asked for (16 rays a warp, 128 a tile, with remainders) nor on its place among
them; random parameters, origins inside and outside of
the scene, zero and tiny directions, and the table's dense and hashed levels."""
import numpy as np
import pytest

import proposer_oracle as PO
from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu

N = 5000


@pytest.fixture(scope="module", params=[9, 128, 300])
def proposer(rtc, request):
    dev = rtc.Device(b"")
    sc = rtc.Scene(dev)
    sc.add_mesh(*W.gaussian_soup(20000, seed=3))
    sc.commit()
    p = rtc.Proposer(sc, seed=1, max_treelets=request.param)
    p.set_params(PO.random_params(seed=5))
    yield p
    p.release()
    sc.release()
    dev.release()


@pytest.fixture(scope="module")
def rays():
    rng = np.random.default_rng(11)
    d = rng.normal(size=(N, 3))
    d[::97] = 0.0
    d[1::97] *= 1e-30
    return R.make_rays(rng.uniform(-0.5, 1.5, (N, 3)), d)


@pytest.mark.parametrize("count", [1, 15, 16, 17, 127, 129, 2049])
def test_prefix_and_order(proposer, rays, count):
    whole = proposer.predict(rays)
    assert (proposer.predict(rays[:count]) == whole[:count]).all()
    perm = np.random.default_rng(count).permutation(N)
    assert (proposer.predict(rays[perm]) == whole[perm]).all()
