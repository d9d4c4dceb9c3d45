"""The sort of small inputs (one CTA up to 4096 keys, tiles of 1024 keys up to 2^18)
against numpy's stable sort and, for the 32-bit keys of a build, against the 64-bit
keys of the same triangles as a batched scene of one batch: sizes around a warp, a
row of the CTA and the rules' lines, few distinct keys (ties keep their order), and
constant digits."""
import numpy as np
import pytest

from rtcgb import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 1023, 1025, 4095, 4096, 4097, 16_385, 262_144, 262_145]


@pytest.mark.parametrize("n", SIZES)
def test_pairs(rtc, n):
    rng = np.random.default_rng(n)
    vals = rng.permutation(n).astype(np.uint32)
    for keys in (rng.integers(0, 2**64, n, dtype=np.uint64), rng.integers(0, 5, n).astype(np.uint64) << np.uint64(37),
                 np.full(n, 2**63 + 5, np.uint64), np.arange(n, 0, -1).astype(np.uint64)):
        order = np.argsort(keys, kind="stable")
        k, v = rtc.radix_sort_pairs(keys, vals)
        assert (k == keys[order]).all() and (v == vals[order]).all()


@pytest.mark.parametrize("n", SIZES)
def test_build_keys(rtc, n):
    soup = W.gaussian_soup(n, seed=n)
    ties = (np.repeat(soup[0][:3], n, 0).reshape(3, n, 3).transpose(1, 0, 2).reshape(-1, 3).copy(),
            np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))  # n times one triangle
    for mesh in (soup, ties) if n <= 5000 else (soup,):
        out = []
        for batched in (False, True):
            dev = rtc.Device(b"gpu.morton_bits=30")
            sc = rtc.Scene(dev)
            sc.set_batched(batched)
            sc.add_mesh(*mesh)
            sc.commit()
            nodes, tris = sc.bvh()
            out.append((nodes.tobytes(), tris.tobytes()))
            sc.release()
            dev.release()
        assert out[0] == out[1]
