"""Traversal stacks above the 48 KB of shared memory that a kernel may have
without asking: contexts of different needs side by side, and scenes whose
worst-case stack fits in no block's shared memory.
"""
import numpy as np
import pytest

import oracle
from vkpathtracer_b200 import native, scenes
from vkpathtracer_b200.tracer import BatchRenderer, CudaPathTracer, material_params

pytestmark = pytest.mark.gpu


def deep_scene(per_axis, glass=False):
    """Triangles at distances of 2.1^k from the origin along three axes: each
    midpoint split takes one off, so the reference's tree is about as deep as it
    has triangles."""
    v = []
    for a in range(3):
        for k in range(per_axis):
            d = 2.1 ** (k - per_axis // 2 + 8)
            for p in ((-1.0, -1.0), (1.0, -1.0), (0.0, 1.0)):
                c = np.zeros(3)
                c[a], c[(a + 1) % 3], c[(a + 2) % 3] = d, p[0], p[1]
                v.append(c)
    sc = scenes.cornell_box(seed=4)
    sc.vertices = np.ascontiguousarray(v, np.float32)
    sc.indices = np.arange(len(v), dtype=np.uint32).reshape(-1, 3)
    sc.instances = np.array([[0, sc.indices.shape[0], 0]], np.uint32)
    sc.materials = sc.materials.copy()
    if glass:
        sc.materials[0, 7:16] = (5, 0.0, 1.5, 0.9, 0.0, 0.0, 0.0, 1.0, 0.0)
    sc.camera = scenes.Camera(position=(0.4, 0.3, -0.2), target=(8.0, 0.4, 0.1))
    return sc


def settings():
    return scenes.RenderSettings(width=24, height=16, spp=2, max_depth=3, seed=5)


def tracer(sc, **kw):
    t = CudaPathTracer(bvh="reference", **kw)
    assert t.configure(settings()) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
    return t


def rays():
    r = np.random.RandomState(3)
    d = r.normal(size=(4001, 3))
    d[:, 0] += 3.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(np.concatenate([r.uniform(-0.5, 0.5, d.shape), d], 1), np.float32)


def frame(t):
    assert t.reset_accumulation()
    t.render_frame(0, 2)
    t.synchronize()
    return t.film()[0]


def test_contexts_with_different_stacks_side_by_side():
    """The context with the larger stack runs again after one with a smaller."""
    sc, q = deep_scene(30), rays()
    rp, rt, _, _ = oracle.load("port").intersect(sc, q, threads=4)
    with tracer(sc, block_size=256, stack_depth=1) as plain, tracer(sc, block_size=256, stack_depth=64) as large, \
            tracer(sc, block_size=256, stack_depth=32) as small:
        assert large.accel_info()["stack_required"] >= 64
        film = frame(plain)
        for t in (large, small, large, small, plain):
            p, tt = t.trace_rays(q)
            assert np.array_equal(p, rp) and np.array_equal(tt.view(np.uint32), rt.view(np.uint32))
            assert np.array_equal(frame(t).view(np.uint32), film.view(np.uint32))


@pytest.mark.parametrize("mode", ["loop", "persistent"])
def test_batches_with_different_stacks_side_by_side(mode):
    sc = deep_scene(30)
    films = []
    with BatchRenderer(bvh="reference") as a, BatchRenderer(bvh="reference") as b:
        for r in (a, b):
            r.add_job(sc, settings())
        for r, depth in ((a, 64), (b, 32), (a, 64), (b, 1)):
            r.run(mode, block_size=256, stack_depth=depth)
            films.append(r.film(0)[0].copy())
    assert all(np.array_equal(films[0].view(np.uint32), f.view(np.uint32)) for f in films)


def test_deep_glass_scene():
    """Transmissive shadow queries spill their stacks like all others.  Only next
    to SDF primitives they run in a kernel that holds them whole."""
    sc = deep_scene(60, glass=True)
    with tracer(sc, block_size=256) as t, tracer(sc, block_size=32) as other:
        assert t.accel_info()["stack_required"] * 256 * 8 > 227 * 1024
        assert np.array_equal(frame(t).view(np.uint32), frame(other).view(np.uint32))
    sc.sdf = scenes.sdf_gallery(seed=3).sdf
    with tracer(sc, block_size=256) as t:
        with pytest.raises(native.VkptcError) as e:
            t.render_frame(0, 1)
        assert e.value.code == native.UNSUPPORTED


def test_adjoint_forward_with_a_stack_too_large_for_its_wavefront():
    """More paths than the per-path kernel has threads take the renderer's launch
    shape; where that does not fit, a path per thread."""
    sc, side = deep_scene(60), 320
    st = scenes.RenderSettings(width=side, height=side, spp=1, max_depth=3, seed=5)
    out = []
    for kw in ({}, dict(block_size=256, stack_depth=1024)):
        with CudaPathTracer(bvh="reference", **kw) as t:
            assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
            assert t.accel_info()["stack_required"] * 256 * 8 > 227 * 1024
            t.adjoint_setup(1, np.full((side, side, 3), 0.25, np.float32))
            loss, image = t.forward(material_params(sc.materials), image=True)
            out.append((loss, image, t.backward()))
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))
