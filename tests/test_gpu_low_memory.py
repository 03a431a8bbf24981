"""Default waves and pools where they do not fit: a frame, a batch and an adjoint
forward go on with smaller ones (the film does not depend on their size) or, the
forward, with a path per thread; sizes that the caller asked for are not changed.
"""
import numpy as np
import pytest

from vkpathtracer_b200 import native, scenes
from vkpathtracer_b200.tracer import BatchRenderer, CudaPathTracer, material_params

pytestmark = pytest.mark.gpu

SIDE = 1024
MIB = 1 << 20


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


class Filled:
    """All of the device's free memory but `leave` bytes taken."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        self.block = torch.empty(max(0, free - self.leave) // MIB * MIB, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch
        self.block = None
        torch.cuda.empty_cache()


def box_tracer(st, **kw):
    sc = scenes.cornell_box(seed=4)
    t = CudaPathTracer(**kw)
    assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
    return t


def test_frame():
    st = scenes.RenderSettings(width=SIDE, height=SIDE, spp=16, max_depth=3, seed=9)   # 2^24 paths: 2.35 GB
    with box_tracer(st, wave_paths=1 << 20) as t:
        t.render_frame(0, st.spp)
        t.synchronize()
        ref = t.film()[:2]
    with box_tracer(st) as t, box_tracer(st, wave_paths=1 << 24) as asked, Filled(1024 * MIB):
        for _ in range(2):
            assert t.reset_accumulation()
            t.render_frame(0, st.spp)
            t.synchronize()
            film = t.film()[:2]
            assert np.array_equal(bits(film[0]), bits(ref[0])) and np.array_equal(film[1], ref[1])
        with pytest.raises(native.VkptcError) as e:
            asked.render_frame(0, st.spp)
        assert e.value.code == native.ALLOC_FAILED
        assert asked.reset_accumulation()   # the context stays usable
        asked.render_frame(0, 1)
        asked.synchronize()


def test_batch():
    st = scenes.RenderSettings(width=SIDE, height=SIDE, spp=8, max_depth=3, seed=9)   # 2^23 paths: 2.1 GB
    with BatchRenderer() as b:
        b.add_job(scenes.cornell_box(seed=4), st)
        b.run("plain")
        ref = b.film(0)
        with Filled(1024 * MIB):
            for _ in range(2):
                stats = b.run("loop")
                film = b.film(0)
                assert np.array_equal(bits(film[0]), bits(ref[0])) and np.array_equal(film[1], ref[1])
                assert 1 << 21 <= stats["pool_paths"] < 1 << 23
            with pytest.raises(native.VkptcError) as e:
                b.run("loop", pool_paths=1 << 24)
            assert e.value.code == native.ALLOC_FAILED
        assert b.run("loop")["pool_paths"] == 1 << 23


def test_adjoint_forward():
    """2^19 paths: 256 MiB of vertex records and 70 MiB of wave."""
    sc, st = scenes.inverse_box_scene(), scenes.inverse_settings(256, 256, 8)
    params, target = material_params(sc.materials), np.full((256, 256, 3), 0.25, np.float32)
    out = []
    for leave in (None, 300 * MIB):
        with CudaPathTracer(bvh="reference") as t:
            assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
            t.adjoint_setup(8, target)
            if leave is None:
                loss, image = t.forward(params, image=True)
            else:
                with Filled(leave):
                    loss, image = t.forward(params, image=True)
            out.append((loss, image, t.backward()))
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(bits(a), bits(b))
