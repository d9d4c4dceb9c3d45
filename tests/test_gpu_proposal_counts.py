"""proposal_hits of an any-hit query counts the rays whose first hit, in the order of
the ray's own traversal, lies in a proposed subtree.  That depends on the ray alone, so
the count must be the same for every run and for every order of the rays (which
decide with whose leaves a ray's are tested in one batch)."""
import numpy as np
import pytest

import proposer_oracle as PO
from rtcgb import rays as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("treelets,tris,size", [(8, 2000, 0.3), (64, 20_000, 0.1), (1024, 100_000, 0.03)])
def test_any_hit_count_does_not_depend_on_batches(rtc, treelets, tris, size):
    dev = rtc.Device(b"")
    rng = np.random.default_rng(7)
    # large triangles: a ray meets several, in proposed subtrees and outside of them
    v = rng.uniform(0.0, 1.0, (tris, 1, 3)) + rng.normal(size=(tris, 3, 3)) * size
    sc = rtc.Scene(dev)
    sc.add_mesh(v.reshape(-1, 3).astype(np.float32), np.arange(3 * tris, dtype=np.uint32).reshape(-1, 3))
    sc.commit()
    prop = rtc.Proposer(sc, seed=1, max_treelets=treelets)
    prop.set_params(PO.random_params(seed=5))
    n = 200_000
    rays = R.make_rays(rng.uniform(0.0, 1.0, (n, 3)), rng.normal(size=(n, 3)), tfar=3.0)
    counts = set()
    for k in range(6):
        work = rays[rng.permutation(n) if k % 2 else np.arange(n)]
        prop.occluded(work)
        assert (work["tfar"] < 0).any()
        counts.add(rtc.last_query_stats()["proposal_hits"])
    assert len(counts) == 1 and min(counts) > 0, counts
    prop.release()
    sc.release()
    dev.release()
