"""Device pointers of ray queries: the kernel reads rays as pairs of floats, so
an array that starts on an odd float is refused before a launch."""
import numpy as np
import pytest

from vkpathtracer_b200 import native, scenes
from vkpathtracer_b200.tracer import CudaPathTracer

pytestmark = pytest.mark.gpu


def test_alignment_is_checked_on_the_host():
    import torch
    sc, n = scenes.cornell_box(seed=4), 333
    r = np.random.RandomState(2)
    rays = np.concatenate([r.uniform(-0.4, 0.4, (n, 3)) + (0.0, 0.5, 0.0), r.normal(size=(n, 3))], 1).astype(np.float32)
    buf = torch.zeros(6 * n + 8, dtype=torch.float32, device="cuda")
    out = torch.zeros((2, n + 8), dtype=torch.int32, device="cuda")
    with CudaPathTracer() as t:
        assert t.configure(scenes.RenderSettings(width=8, height=8, spp=1))
        assert t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
        prim, dist = t.trace_rays(rays)
        for skip in (0, 1, 2, 3, 4):   # floats before the first ray
            buf[skip:skip + 6 * n] = torch.from_numpy(rays.reshape(-1)).cuda()
            torch.cuda.synchronize()
            call = lambda d_rays, d_prim, d_t: t.trace_rays_device(d_rays, 0, n, native.QUERY_CLOSEST, d_prim, d_t)
            args = [buf.data_ptr() + 4 * skip, out[0].data_ptr() + 4 * skip, out[1].data_ptr() + 4 * skip]
            if skip % 2:
                with pytest.raises(native.VkptcError) as e:
                    call(*args)
                assert e.value.code == native.INVALID_ARGUMENT
                continue
            call(*args)
            t.synchronize()
            got = out[:, skip:skip + n].cpu().numpy()
            assert np.array_equal(got[0].view(np.uint32), prim)
            assert np.array_equal(got[1].view(np.uint32), dist.view(np.uint32))
            for k in (1, 2):
                with pytest.raises(native.VkptcError) as e:
                    call(*[a + 2 * (j == k) for j, a in enumerate(args)])
                assert e.value.code == native.INVALID_ARGUMENT
