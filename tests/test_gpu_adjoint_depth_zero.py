"""A depth of 0 has no vertices: a black image, no gradient, on both sides of the
line from which the forward runs as a wavefront."""
import numpy as np
import pytest

from vkpathtracer_b200 import scenes
from vkpathtracer_b200.tracer import CudaPathTracer, material_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [24, 400])
def test_black_image_and_no_gradient(side):
    sc, st = scenes.inverse_box_scene(), scenes.inverse_settings(side, side, 2)
    st.max_depth = 0
    with CudaPathTracer(bvh="reference") as t:
        assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
        t.adjoint_setup(2, np.full((side, side, 3), 0.5, np.float32))
        for _ in range(2):
            loss, image = t.forward(material_params(sc.materials), image=True)
            assert loss == 0.25 and not np.any(image) and not np.any(t.backward())
        assert not np.any(t.adjoint_samples()[0])
