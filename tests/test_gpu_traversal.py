"""The wide-BVH traversal where its box test could go wrong: direction
components of zero and around the reference's parallel limit (1e-4), rays along
the axes and through box faces, scenes far from the origin and of very
different scales, huge and tiny direction components, and traversal stacks that
spill out of shared memory.  Closest-hit ids and distances are the oracle's bit
for bit (the device's box test only culls); any-hit is its "closest t < tmax".

Two limits of that statement, which any box test with other rounding than the
reference's has.  The probes aim at vertices, where several triangles report
distances some ulps apart, and a grazing triangle (|det| near 1e-4) can report
one outside its box, so which of them is visited decides:
  * beyond coordinates of about 200 the reference's 1e-4 box padding is a few
    ulps, and its own rounding culls such triangles: there one probe in 500 may
    name another triangle, its distance within 1e-5 of the oracle's;
  * a bound 1e-4 above the closest distance may cull the grazing triangle's box:
    one any-hit probe in 2000 may then report no occluder (unbounded any-hit is
    exact).
"""
import numpy as np
import pytest

import oracle
from vkpathtracer_b200 import native, scenes
from vkpathtracer_b200.tracer import CudaPathTracer

pytestmark = pytest.mark.gpu


def probe_rays(sc, n, seed):
    """Rays from around the scene at its vertices, a part of them with
    components set to 0, to values around 1e-4, or aligned with an axis."""
    r = np.random.RandomState(seed)
    v = np.asarray(sc.vertices, np.float64)
    mid, half = 0.5 * (v.min(0) + v.max(0)), 0.5 * (v.max(0) - v.min(0)).max()
    o = mid + r.uniform(-2.0, 2.0, (n, 3)) * half
    target = v[r.randint(0, v.shape[0], n)]
    d = target - o
    d /= np.maximum(1e-12, np.linalg.norm(d, axis=1, keepdims=True))
    kind = r.randint(0, 6, n)
    axis = r.randint(0, 3, n)
    rows = np.arange(n)
    small = np.array([0.0, -0.0, 1e-30, -1e-12, 9.9e-5, -1.01e-4])
    k = kind == 1   # one tiny component, from a point level with the target
    d[rows[k], axis[k]] = small[r.randint(0, small.size, k.sum())]
    o[rows[k], axis[k]] = target[rows[k], axis[k]]
    k = kind == 2   # along an axis, through a vertex or near one
    d[k] = 0.0
    d[rows[k], axis[k]] = r.choice([-1.0, 1.0], k.sum())
    off = r.choice([0.0, 1e-5, 1e-3], (k.sum(), 3)) * half
    o[k] = target[k] + off - d[k] * 3.0 * half
    k = kind == 3   # unnormalised directions
    d[k] *= 10.0 ** r.uniform(-3.0, 3.0, (k.sum(), 1))
    return np.ascontiguousarray(np.concatenate([o, d], axis=1), np.float32)


def tracer(sc, **kw):
    t = CudaPathTracer(**kw)
    assert t.configure(scenes.RenderSettings(width=8, height=8, spp=1))
    assert t.load_scene_snapshot(sc)
    assert t.build_or_update_acceleration()
    return t


def check(sc, rays, test="mt", **kw):
    o = oracle.load("port")
    with o.triangle_test("watertight" if test == "watertight" else "mt"):
        rp, rt, _, _ = o.intersect(sc, rays, threads=8)
    tmax = np.where(np.isfinite(rt), rt * np.float32(1.0001), np.float32(50.0)).astype(np.float32)
    with tracer(sc, triangle_test=test, **kw) as t:
        p, tt = t.trace_rays(rays)
        a, _ = t.trace_rays(rays, mode=native.QUERY_ANY, tmax=tmax)
        u, _ = t.trace_rays(rays, mode=native.QUERY_ANY)
    assert np.array_equal(u.astype(bool), np.isfinite(rt))
    differ = (p != rp) | (tt.view(np.uint32) != rt.view(np.uint32))
    far = np.abs(sc.vertices).max() > 200.0
    assert differ.sum() <= (p.size // 500 if far else 0), f"{differ.sum()} of {p.size} hits differ"
    assert np.allclose(tt[differ], rt[differ], rtol=1e-5, atol=0.0)
    wrong = a.astype(bool) != (np.isfinite(rt) & (rt < tmax))
    assert not np.any(a[wrong]) and wrong.sum() <= p.size // 2000, f"{wrong.sum()} of {p.size} any-hit answers differ"
    return rp


@pytest.mark.parametrize("test", ["mt", "watertight"])
@pytest.mark.parametrize("bvh", ["reference", "sah"])
@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (16.0, 0.0), (16.0, 300.0), (250.0, -100.0)])
def test_axis_and_scale_probes(scale, offset, bvh, test):
    sc = scenes.displaced_sphere(40, scale=scale, seed=5)
    sc.vertices = np.ascontiguousarray(sc.vertices + np.array([offset, 0.5 * offset, -offset], np.float32))
    prim = check(sc, probe_rays(sc, 20011, 7), test=test, bvh=bvh)
    if scale >= 16.0:
        assert np.mean(prim != 0xFFFFFFFF) > 0.3   # the probes do hit


@pytest.mark.parametrize("bvh", ["reference", "sah"])
@pytest.mark.parametrize("stack_depth", [1, 2, 3, 5])
@pytest.mark.parametrize("n", [1, 31, 4097])
def test_spilled_stacks(n, stack_depth, bvh):
    sc = scenes.sphere_field(4, 15, 18, seed=3, n_lights=2)
    check(sc, probe_rays(sc, n, 11 + n), bvh=bvh, stack_depth=stack_depth)


def test_box_faces_and_root_leaf():
    box = scenes.cornell_box(seed=4)
    check(box, probe_rays(box, 6007, 3))
    one = scenes.cornell_box(seed=4)   # one triangle: the root is a leaf
    one.indices = np.ascontiguousarray(one.indices[:1])
    one.instances = np.array([[0, 1, 0]], np.uint32)
    check(one, probe_rays(one, 1009, 3))


def test_non_finite_rays_end_and_hit_nothing():
    sc = scenes.sphere_field(3, 15, 18, seed=3, n_lights=2)
    rays = probe_rays(sc, 64, 5)
    bad = np.array([np.nan, np.inf, -np.inf], np.float32)
    for k in range(36):
        rays[k, k % 6] = bad[k // 12]
    with tracer(sc, bvh="sah") as t:
        p, tt = t.trace_rays(rays)
    assert np.all(p[:12] == 0xFFFFFFFF) and np.all(np.isinf(tt[:12]))
    rp, rt, _, _ = oracle.load("port").intersect(sc, rays[36:], threads=1)
    assert np.array_equal(p[36:], rp) and np.array_equal(tt[36:].view(np.uint32), rt.view(np.uint32))


@pytest.mark.parametrize("n_lat,n_lon", [(2, 3), (3, 4), (3, 6), (4, 11), (5, 8), (5, 9), (8, 9), (9, 32), (17, 33), (33, 40)])
def test_sah_trees_at_subtree_and_chunk_edges(n_lat, n_lon):
    """SAH trees whose sizes straddle the leaf limit (2), the ten planes and the
    64 primitives of a warp's subtree, and the 512 positions of a binning block:
    6, 16, 24, 66, 64, 72, 126, 512, 1056 and 2560 triangles, and three copies
    of each (coinciding centroids, every hit a tie).  Every triangle is in the
    tree once, and rays aimed inside triangles hit what the oracle's hit."""
    one = scenes.sphere_field(1, n_lat, n_lon, seed=2, n_lights=1)
    tri = np.ascontiguousarray(one.indices[:2 * (n_lat - 1) * n_lon])
    r = np.random.RandomState(n_lat)
    for copies in (1, 3):
        sc = scenes.sphere_field(1, n_lat, n_lon, seed=2, n_lights=1)
        sc.vertices = np.ascontiguousarray(sc.vertices * np.float32(16.0))
        sc.indices = np.ascontiguousarray(np.concatenate([tri] * copies))
        sc.instances = np.array([[0, sc.indices.shape[0], 0]], np.uint32)
        w = r.dirichlet((2.0, 2.0, 2.0), 3001)
        target = np.einsum("nk,nkc->nc", w, sc.vertices[tri[r.randint(0, tri.shape[0], 3001)]].astype(np.float64))
        o = r.uniform(-60.0, 60.0, (3001, 3))
        rays = np.ascontiguousarray(np.concatenate([o, target - o], axis=1), np.float32)
        rays[:, 3:] /= np.linalg.norm(rays[:, 3:], axis=1, keepdims=True)
        rp, rt, _, _ = oracle.load("port").intersect(sc, rays, threads=8)
        with tracer(sc, bvh="sah") as t:
            p, tt = t.trace_rays(rays)
            rec = t.read_accel(native.ACCEL_TRIANGLES).reshape(-1, 12)
        assert np.array_equal(np.sort(rec[:, 9]), np.arange(sc.indices.shape[0]))
        assert np.array_equal(p, rp) and np.array_equal(tt.view(np.uint32), rt.view(np.uint32))


@pytest.mark.parametrize("block_size", [0, 32, 256])
@pytest.mark.parametrize("extra", [-1, 0, 1, 33])
def test_ray_counts_around_one_per_thread(extra, block_size):
    """Calls of at most one ray per resident thread are spread over the warps
    without a query counter; the count where that ends depends on the device, so
    counts around every multiple of its threads per block and SM are tried."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sc = scenes.cornell_box(seed=4)
    n = sms * 1024 + extra
    rays = probe_rays(sc, n, 9)
    rp, rt, _, _ = oracle.load("port").intersect(sc, rays, threads=8)
    with tracer(sc, block_size=block_size) as t:
        for k in (n, sms * 32 + extra, 5 * sms + extra):
            p, tt = t.trace_rays(rays[:k])
            assert np.array_equal(p, rp[:k]) and np.array_equal(tt.view(np.uint32), rt[:k].view(np.uint32))
