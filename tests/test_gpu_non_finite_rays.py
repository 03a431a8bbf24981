"""Rays with a NaN or infinite component hit nothing, in any component and beside
finite rays of the same warp, which hit what the oracle's do."""
import numpy as np
import pytest

import oracle
from tests.test_gpu_traversal import probe_rays, tracer
from vkpathtracer_b200 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("test", ["mt", "watertight"])
@pytest.mark.parametrize("bvh", ["reference", "sah"])
def test_every_component(bvh, test):
    sc = scenes.sphere_field(3, 15, 18, seed=3, n_lights=2)
    n = 1024
    rays = probe_rays(sc, n, 5)
    r = np.random.RandomState(1)
    bad = np.array([np.nan, np.inf, -np.inf], np.float32)
    rows = np.arange(0, n, 2)
    rays[rows, rows // 2 % 6] = bad[rows // 12 % 3]
    rays[rows[::3], r.randint(0, 6, rows[::3].size)] = bad[r.randint(0, 3, rows[::3].size)]
    finite = np.ones(n, bool)
    finite[rows] = False
    o = oracle.load("port")
    with o.triangle_test(test):
        rp, rt, _, _ = o.intersect(sc, np.ascontiguousarray(rays[finite]), threads=4)
    with tracer(sc, bvh=bvh, triangle_test=test) as t:
        p, tt = t.trace_rays(rays)
        answers = [t.trace_rays(rays, mode=native.QUERY_ANY, tmax=tm)[0]
                   for tm in (None, np.full(n, 7.0, np.float32), np.full(n, np.nan, np.float32))]
    assert np.all(p[~finite] == 0xFFFFFFFF) and np.all(np.isposinf(tt[~finite]))
    assert np.array_equal(p[finite], rp) and np.array_equal(tt[finite].view(np.uint32), rt.view(np.uint32))
    for a in answers:
        assert not np.any(a[~finite])
    assert np.array_equal(answers[0][finite].astype(bool), np.isfinite(rt)) and not np.any(answers[2])
