"""Traversal counters of the wavefront next to the persistent driver's, which
tests SDF occlusion where it shades and queues only what is left."""
import pytest

from vkpathtracer_b200 import scenes
from vkpathtracer_b200.tracer import BatchRenderer, CudaPathTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["box", "sdf"])
def test_ray_counts_equal_the_persistent_drivers(kind):
    sc = scenes.cornell_box(seed=2) if kind == "box" else scenes.sdf_gallery(seed=3)
    st = scenes.RenderSettings(width=61, height=47, spp=4, max_depth=6, seed=23)
    with CudaPathTracer(collect_stats=True) as t:
        assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
        t.render_frame(0, st.spp)
        t.synchronize()
        wave, tests = t.traversal_stats(), t.read_counters()["shadow_tests"]
    with BatchRenderer(collect_stats=True) as b:
        b.add_job(sc, st)
        persistent = b.run("persistent")
    assert wave["rays"] == persistent["ext_rays"]
    assert wave["shadow_rays"] == persistent["shadow_queries"]
    assert (wave["shadow_rays"] == tests) == (kind == "box")   # SDF primitives occlude some
