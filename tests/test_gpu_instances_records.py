"""Scenes with instances: the kernels for few and for many rays, on aligned and unaligned
records, against the oracle's instance restatement.  The instances overlap, so leaf
groups are interrupted by an instance and resumed, several deep on the stack."""
import numpy as np
import pytest

from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu

MOST_FEW = 3 << 18  # rays that the few-ray kernel takes at most
CHECKED = 20_000    # rays that the oracle traces


@pytest.fixture(scope="module")
def scenes(rtc, oracle):
    dev = rtc.Device(b"")
    rng = np.random.default_rng(29)
    meshes = [W.gaussian_soup(3000, seed=1), W.heightfield(12, seed=2)]
    children, ochildren = [], []
    for v, i in meshes:
        c = rtc.Scene(dev)
        c.add_mesh(v, i)
        c.commit()
        children.append(c)
        ochildren.append(oracle.OracleScene([(0, v, i)]))
    top = rtc.Scene(dev)
    own = W.gaussian_soup(500, seed=5)
    top.add_mesh(*own)
    insts = []
    for k in range(40):
        m = np.diag(rng.uniform(0.3, 0.9, 3)) @ np.linalg.qr(rng.normal(size=(3, 3)))[0]
        x = np.concatenate([m[:, 0], m[:, 1], m[:, 2], rng.uniform(0.0, 0.4, 3)]).astype(np.float32)
        insts.append((ochildren[k % 2], x, top.add_instance(children[k % 2], x)))
    top.commit()
    yield top, oracle.OracleScene([(0, *own)]), insts
    for s in (top, *children):
        s.release()
    dev.release()


def _strided(recs, stride):
    buf = np.zeros((recs.shape[0], stride), np.uint8)
    buf[:, :recs.itemsize] = recs.view(np.uint8).reshape(-1, recs.itemsize)
    return buf


@pytest.mark.parametrize("stride", [80, 84, 96])
@pytest.mark.parametrize("count", [1, 33, CHECKED, MOST_FEW, MOST_FEW + 1])
def test_records_match_oracle(oracle, scenes, stride, count):
    top, otop, insts = scenes
    rays = W.sphere_rays(count, seed=31)
    buf = _strided(rays, stride)
    top.intersect_ptr(buf.ctypes.data, count, stride)
    n = min(count, CHECKED)
    g = np.ascontiguousarray(buf[-n:, :80]).view(R.RAYHIT_DTYPE).reshape(-1)
    r = rays[-n:].copy()
    oracle.instanced(otop, insts, r)
    same = (g["geomID"] == r["geomID"]) & (g["primID"] == r["primID"]) & (g["instID"] == r["instID"])
    # different triangles at exactly the same distance are ties of the visiting order
    tie = ~same & (g["tfar"].view(np.uint32) == r["tfar"].view(np.uint32))
    assert (same | tie).all() and tie.sum() <= 10
    assert R.hits_equal_bits(g[same], r[same]).all()
    assert not buf[:, 80:].any()
    sh = np.zeros(count, R.RAY_DTYPE)
    for f in R.RAY_DTYPE.names:
        sh[f] = rays[f]
    sh["tfar"] = 0.3
    buf = _strided(sh, stride)
    top.occluded_ptr(buf.ctypes.data, count, stride)
    g = np.ascontiguousarray(buf[-n:, :48]).view(R.RAY_DTYPE).reshape(-1)
    r = sh[-n:].copy()
    oracle.instanced(otop, insts, r, anyhit=True)
    assert (g.view(np.uint8) == r.view(np.uint8)).all()
