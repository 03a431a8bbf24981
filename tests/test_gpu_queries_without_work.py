"""More queries than a launch has threads of which many end when they are loaded
(a scene without triangles, a bound of zero, a query that an SDF primitive
occludes): the ones after them are still claimed."""
import numpy as np
import pytest

import oracle
from tests.test_gpu_traversal import probe_rays, tracer
from vkpathtracer_b200 import native, scenes
from vkpathtracer_b200.tracer import BatchRenderer, CudaPathTracer, RenderTile

pytestmark = pytest.mark.gpu

N = 1_200_007   # several times the 303,104 threads of a launch on 148 SMs


def test_no_triangles():
    sc = scenes.cornell_box(seed=4)
    rays = probe_rays(sc, N, 3)
    sc.indices, sc.instances = np.zeros((0, 3), np.uint32), np.zeros((0, 3), np.uint32)
    with tracer(sc) as t:
        p, tt = t.trace_rays(rays)
        a, _ = t.trace_rays(rays, mode=native.QUERY_ANY)
    assert np.all(p == 0xFFFFFFFF) and np.all(np.isposinf(tt)) and not np.any(a)


@pytest.mark.parametrize("steps", [0, 8 | 16 << 16])   # with a refill threshold, too
def test_bounds_of_zero(steps):
    sc = scenes.cornell_box(seed=4)
    rays = probe_rays(sc, N, 3)
    rp, rt, _, _ = oracle.load("port").intersect(sc, rays[-2000:], threads=4)
    tmax = np.zeros(N, np.float32)
    tmax[-2000:] = np.inf
    with tracer(sc, steps=steps) as t:
        a, _ = t.trace_rays(rays, mode=native.QUERY_ANY, tmax=tmax)
    assert not np.any(a[:-2000]) and np.array_equal(a[-2000:].astype(bool), np.isfinite(rt))


def test_sdf_scene_without_triangles():
    """The frame in one wave, in small tiles and by the batch drivers."""
    sc = scenes.sdf_complexity()
    assert sc.triangle_count == 0
    st = scenes.RenderSettings(width=640, height=480, spp=4, max_depth=4, seed=11)
    films = []
    for tiles in (False, True):
        with CudaPathTracer() as t:
            assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
            if tiles:   # waves of fewer paths than a launch has threads
                for y in range(0, st.height, 60):
                    for s in range(st.spp):
                        assert t.render_tile(RenderTile(0, y, st.width, 60, s))
            else:
                t.render_frame(0, st.spp)
            t.synchronize()
            films.append(t.film()[0])
    with BatchRenderer() as b:
        b.add_job(sc, st)
        for mode in ("loop", "persistent"):
            b.run(mode)
            films.append(b.film(0)[0])
    for f in films[1:]:
        assert np.array_equal(films[0].view(np.uint32), f.view(np.uint32))
