"""Sort keys of scenes side by side: with up to 1,023 scenes they are 40 bits wide, the
invalid triangles' all ones.  Around that line the valid triangles of every scene, and
no others, must come out, alike from the host-driven and the replayed build and in
either key width's grouping, with triangles at the key space's far corner and invalid
ones in every scene."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(k):
    """Three triangles: one spread over the scene box, one in its last corner, one invalid."""
    v = np.array([[-1, -1, -1], [1, 1, 1], [0, 1, 0], [1, 1, 1], [1, 1, 1], [1, 1, 1], [np.nan, 0, 0], [0, 1, 0],
                  [0, 0, 1]], np.float32)
    v[:3] *= np.float32(1 - k * 1e-5)
    return v, np.arange(9, dtype=np.uint32).reshape(3, 3)


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("scenes", [1, 2, 1022, 1023, 1024])
def test_valid_triangles_of_every_scene(rtc, scenes, bits):
    out = []
    for graph in (0, 1):
        dev = rtc.Device(f"gpu.morton_bits={bits},gpu.graph_rebuild={graph}".encode())
        sc = rtc.Scene(dev)
        sc.set_batched(True)
        for k in range(scenes):
            sc.add_mesh(*_mesh(k))
        for _ in range(4):
            sc.commit()
            nodes, tris = sc.bvh()
            out.append((nodes.tobytes(), tris.tobytes()))
        assert len(tris) == 2 * scenes
        sc.release()
        dev.release()
    assert all(x == out[0] for x in out)
