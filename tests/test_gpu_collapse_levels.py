"""The collapse of captured builds (all levels in one launch, offsets from sums that the
CTAs read of each other) must give the host-driven build's nodes and triangles byte for
byte: levels of one node, of up to 32 and of more nodes a CTA, both CTA sizes, leaves of
one to four triangles, children with equal slot costs, and scenes side by side."""
import numpy as np
import pytest

from rtcgb import workloads as W

pytestmark = pytest.mark.gpu


def _grid(n):
    """Triangles on a square grid: boxes around a node's centre tie in their slot costs."""
    side = max(2, int(round((n / 2) ** 0.5)))
    return W.triangle_plane((-1, 0, -1), (2, 0, 0), (0, 0, 2), side, side)


def _commits(rtc, cfg, mesh, count):
    dev = rtc.Device(cfg)
    sc = rtc.Scene(dev)
    sc.set_batched(count > 1)
    for _ in range(count):
        sc.add_mesh(*mesh)
    out = []
    for _ in range(3):  # the third is replayed
        sc.commit()
        nodes, tris = sc.bvh()
        out.append((nodes.tobytes(), tris.tobytes()))
    sc.release()
    dev.release()
    return out


@pytest.mark.parametrize("leaf", [1, 2, 4])
@pytest.mark.parametrize("n,count", [(1, 1), (9, 1), (700, 1), (40_000, 1), (1_100_000, 1), (3, 500), (900, 40)])
def test_replayed_collapse_equals_host_driven(rtc, n, count, leaf):
    for mesh in (W.gaussian_soup(n, seed=n + leaf), _grid(n)):
        ref = _commits(rtc, f"gpu.graph_rebuild=0,gpu.leaf_max={leaf}".encode(), mesh, count)
        got = _commits(rtc, f"gpu.leaf_max={leaf}".encode(), mesh, count)
        assert all(x == ref[0] for x in ref + got)
