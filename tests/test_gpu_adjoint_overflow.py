"""Gradients beyond the range of a float: the slots of the reverse sweep keep an
infinity an infinity."""
import numpy as np
import pytest

from vkpathtracer_b200 import scenes
from vkpathtracer_b200.tracer import CudaPathTracer, material_params

pytestmark = pytest.mark.gpu


def test_infinite_gradient_stays_infinite():
    """Targets near the largest float and lights of 1e8 times their power: the
    image is far below the target, so every albedo's derivative, which carries the
    lights' power, is minus infinity, and every emission's, which does not, is a
    negative number."""
    sc, st = scenes.inverse_box_scene(), scenes.inverse_settings(32, 32, 8)
    sc.lights[:, 6] *= 1e8
    with CudaPathTracer(bvh="reference") as t:
        assert t.configure(st) and t.load_scene_snapshot(sc) and t.build_or_update_acceleration()
        t.adjoint_setup(8, np.full((32, 32, 3), 3e38, np.float32))
        t.forward(material_params(sc.materials))
        g = t.backward().reshape(-1, 7)
    lit = np.any(g[:, :3] != 0.0, axis=1)
    assert lit.sum() > 10 and np.all(np.isneginf(g[lit, :3]))
    seen = np.any(g[:, 4:] != 0.0, axis=1)
    assert seen.sum() > 10 and np.all(np.isfinite(g[:, 4:])) and np.all(g[seen, 4:] < 0.0)
