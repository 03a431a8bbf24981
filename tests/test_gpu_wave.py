"""A wave's slots (8x4 pixel tiles, 32 pixels at a time, all samples of 32
pixels together, the last pixels sample-major) and its merged trace launches:
frames whose sizes straddle the tiles, rendered whole, split into several waves
and pixel by pixel, give the same film bit for bit; transmissive shadow queries
and SDF primitives give the oracle's film.
"""
import numpy as np
import pytest

import oracle
from tests.test_gpu_parity import BIT_EXACT_FRAC, RMSE_REL_TOL, film_report
from vkpathtracer_b200 import scenes
from vkpathtracer_b200.tracer import CudaPathTracer, RenderTile

pytestmark = pytest.mark.gpu


def glass_box():
    """The closed box with one glass and one half-transparent box (no SDF primitives)."""
    sc = scenes.cornell_box(seed=2)
    sc.materials[5, 7:16] = (5, 0.0, 1.5, 0.9, 0.0, 0.0, 0.0, 1.0, 0.0)
    sc.materials[6, 10] = 0.4
    sc.name = "glass_box"
    return sc


def make_scene(kind):
    return {"field": lambda: scenes.sphere_field(3, 10, 12, seed=4, n_lights=2, light_size=1.0, light_height=4.0),
            "glass": glass_box, "sdf": lambda: scenes.sdf_gallery(seed=3),
            "sdf_glass": lambda: scenes.sdf_gallery(seed=3, glass=True)}[kind]()


def render(sc, st, calls, **kw):
    with CudaPathTracer(**kw) as t:
        assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
        assert t.reset_accumulation()
        calls(t)
        t.synchronize()
        film, count, _ = t.film()
        return film, count, t.read_counters()


@pytest.mark.parametrize("kind", ["field", "glass", "sdf", "sdf_glass"])
@pytest.mark.parametrize("w,h", [(1, 1), (7, 3), (8, 4), (9, 5), (31, 1), (33, 2), (4, 9)])
def test_slot_orders_agree(w, h, kind):
    sc = make_scene(kind)
    st = scenes.RenderSettings(width=w, height=h, spp=3, max_depth=5, seed=19)
    whole = render(sc, st, lambda t: t.render_frame(0, st.spp))
    waves = render(sc, st, lambda t: t.render_frame(0, st.spp), wave_paths=2 * w * h)

    def pixels(t):
        for s in range(st.spp):
            for y in range(h):
                assert t.render_tiles([RenderTile(x, y, 1, 1, s) for x in range(w)])

    single = render(sc, st, pixels)
    for other in (waves, single):
        assert np.array_equal(whole[0].view(np.uint32), other[0].view(np.uint32))
        assert np.array_equal(whole[1], other[1])
        for k in ("samples", "rays", "shadow_tests"):
            assert whole[2][k] == other[2][k], k


@pytest.mark.parametrize("kind", ["field", "glass", "sdf", "sdf_glass"])
@pytest.mark.parametrize("depth", [1, 2, 7])
def test_films_match_the_oracle(kind, depth):
    sc = make_scene(kind)
    st = scenes.RenderSettings(width=61, height=47, spp=4, max_depth=depth, seed=23)
    film, count, _ = render(sc, st, lambda t: t.render_frame(0, st.spp))
    ref = oracle.load("port").render(sc, st, per_sample=True)
    r = film_report(film, ref["sum"], ref["samples"], st.spp)
    print(kind, depth, r)
    assert np.array_equal(count, ref["count"])
    assert r["rmse_rel"] < RMSE_REL_TOL and r["bit_exact"] >= BIT_EXACT_FRAC
