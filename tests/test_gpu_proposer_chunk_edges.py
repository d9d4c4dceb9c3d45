"""Proposer inference around the edges of the 128-treelet chunks of the tcgen05 kernel,
with odd and even numbers of chunks and with several 128-ray tiles per CTA (which take
the accumulators in turn): the proposals are those of the mma.sync kernel over the same
treelets, up to ties of the FP32 accumulation order."""
import numpy as np
import pytest

import proposer_oracle as PO
from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu

MANY = 128 * 1600 + 77  # five or six tiles for each of 304 CTAs, the last one ragged


@pytest.fixture(scope="module")
def scenes(rtc):
    devs = [rtc.Device(b""), rtc.Device(b"gpu.proposer=mma")]
    out = []
    for d in devs:
        sc = rtc.Scene(d)
        sc.add_mesh(*W.heightfield(48))
        sc.add_mesh(*W.gaussian_soup(40000, seed=3))
        sc.commit()
        out.append(sc)
    yield out
    for sc in out:
        sc.release()
    for d in devs:
        d.release()


@pytest.mark.parametrize("treelets", [127, 128, 129, 256, 257, 385, 640])
def test_chunk_edges_match_mma_sync(rtc, scenes, treelets):
    params = PO.random_params(seed=13)
    props = [rtc.Proposer(sc, seed=1, max_treelets=treelets) for sc in scenes]
    have = [p.stats()["num_treelets"] for p in props]  # whole subtrees: the budget or a few less
    assert have[0] == have[1] <= treelets and (have[0] + 127) // 128 == (treelets + 127) // 128
    rng = np.random.default_rng(treelets)
    d = rng.normal(size=(MANY, 3))
    rays = R.make_rays(rng.uniform(0.05, 0.95, (MANY, 3)), d / np.linalg.norm(d, axis=1, keepdims=True))
    got = []
    for p in props:
        p.set_params(params)
        got.append(p.predict(rays))
    assert (got[0] < have[0]).all()
    assert (np.sort(got[0], 1) == np.sort(got[1], 1)).all(1).mean() > 0.99
    # proposals from both sides of the last chunk's edge
    edge = (treelets - 1) // 128 * 128
    assert (got[0] >= edge).any() and (edge == 0 or (got[0] < edge).any())
    for p in props:
        p.release()
