"""Clustering with search radius 1: the rounds and the finish that merge at local
minima of the adjacent areas (captured builds) must give the host-driven build's
tree byte for byte, around the sizes of a tile, of a CTA's run and of the one-CTA
finish, with equal areas (ties) and with scenes side by side."""
import numpy as np
import pytest

from rtcgb import workloads as W

pytestmark = pytest.mark.gpu


def _random(n):
    return W.gaussian_soup(n, seed=n)


def _equal(n):
    """A regular row of equal triangles: every adjacent area ties."""
    base = np.array([[0, 0, 0], [0.5, 0, 0], [0, 0.5, 0]], np.float32)
    v = base[None] + np.arange(n, dtype=np.float32)[:, None, None] * np.array([1, 0, 0], np.float32)
    return v.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def _plane(n):
    return W.triangle_plane((0, 0, 0), (1, 0, 0), (0, 1, 0), max(1, n // 64), 32)


def _commits(rtc, cfg, meshes, batched):
    dev = rtc.Device(cfg)
    sc = rtc.Scene(dev)
    if batched:
        sc.set_batched(True)
    for m in meshes:
        sc.add_mesh(*m)
    out = []
    for _ in range(4):  # host-driven, host-driven, replayed, replayed
        sc.commit()
        nodes, tris = sc.bvh()
        out.append((nodes.tobytes(), tris.tobytes()))
    sc.release()
    dev.release()
    return out


@pytest.mark.parametrize("mesh", [_random, _equal, _plane], ids=["random", "equal", "plane"])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 257, 4095, 4097, 8225, 60_000])
def test_replayed_tree_equals_host_driven(rtc, mesh, n):
    ref = _commits(rtc, b"gpu.graph_rebuild=0", [mesh(n)], False)
    got = _commits(rtc, b"", [mesh(n)], False)
    assert all(x == ref[0] for x in ref + got)


@pytest.mark.parametrize("sizes", [(1, 1, 1), (5, 4000, 31, 1, 4097), tuple([3] * 700)], ids=["ones", "mixed", "many"])
def test_batched_scenes(rtc, sizes):
    meshes = [_random(n) if k % 2 else _equal(n) for k, n in enumerate(sizes)]
    ref = _commits(rtc, b"gpu.graph_rebuild=0", meshes, True)
    got = _commits(rtc, b"", meshes, True)
    assert all(x == ref[0] for x in ref + got)
