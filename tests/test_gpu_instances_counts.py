"""Scenes with instances are traced by one of two kernels of the same code, by the number
of rays: the same rays alone (few) and as part of a long stream must give the same bytes,
closest hit and occlusion, aligned and unaligned records, on both sides of the line."""
import numpy as np
import pytest

from rtcgb import rays as R
from rtcgb import workloads as W

pytestmark = pytest.mark.gpu

LINE = 1 << 19


@pytest.mark.parametrize("count", [LINE, LINE + 1])
def test_few_and_many_rays(rtc, count):
    dev = rtc.Device(b"")
    child, top = rtc.Scene(dev), rtc.Scene(dev)
    child.add_mesh(*W.gaussian_soup(3000, seed=1))
    child.commit()
    rng = np.random.default_rng(3)
    for _ in range(20):
        m = np.diag(rng.uniform(0.1, 0.3, 3))
        top.add_instance(child, np.concatenate([m[:, 0], m[:, 1], m[:, 2], rng.uniform(-1, 1, 3)]).astype(np.float32))
    top.commit()
    org, dirs = rng.uniform(-1.5, 1.5, (count, 3)), rng.normal(size=(count, 3))
    for make, query in ((R.make_rayhits, top.intersect), (R.make_rays, top.occluded)):
        many = make(org, dirs)
        few = many[-5000:].copy()
        query(many)
        query(few)
        assert many[-5000:].tobytes() == few.tobytes()
    for s in (top, child):
        s.release()
    dev.release()
