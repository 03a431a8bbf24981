"""The forward's image goes into exactly W x H x 3 floats, also after a larger set-up."""
import ctypes

import numpy as np
import pytest

from vkpathtracer_b200 import native, scenes
from vkpathtracer_b200.tracer import CudaPathTracer, material_params

pytestmark = pytest.mark.gpu


def test_image_after_a_larger_set_up():
    sc = scenes.inverse_box_scene()
    params = np.ascontiguousarray(material_params(sc.materials), np.float32).reshape(-1)
    with CudaPathTracer(bvh="reference") as t:
        for side in (48, 16):
            st = scenes.inverse_settings(side, side, 4)
            assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
            t.adjoint_setup(4)
            out = np.full(3 * 48 * 48, -7.0, np.float32)   # room for the larger image
            loss = ctypes.c_double(0.0)
            rc = t._lib.vkptc_forward(t._ctx, params.ctypes.data, params.size, None, ctypes.byref(loss), out.ctypes.data)
            assert rc == native.OK
            n = 3 * side * side
            assert np.all(out[:n] >= 0.0) and np.all(out[n:] == -7.0)
