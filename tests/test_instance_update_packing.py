"""Instance updates packed for the C call: the same words as field-by-field
assignment gives, and the same refusals."""
import ctypes

import numpy as np
import pytest

from vkpathtracer_b200 import native, tracer


class Library:
    """Keeps the words of the updates it is called with."""

    def vkptc_update_instance_transforms(self, ctx, arr, count):
        self.words = ctypes.string_at(arr, count * ctypes.sizeof(native.InstanceUpdate))
        return native.OK


def update(updates):
    t = tracer.CudaPathTracer.__new__(tracer.CudaPathTracer)
    t._lib, t._ctx = Library(), None
    tracer.CudaPathTracer.update_instance_transforms(t, updates)
    return t._lib.words


def test_words_are_the_fields():
    ups = [{"instance": 7, "flags": 3, "translation": (1, 2.5, -3), "rotation": [0.1, 0.2, 0.3, 0.4], "scale": np.arange(3.0)},
           {"instance": np.uint32(2)}, {"instance": 5, "translation": np.ones(3, np.float32), "scale": (1e39, 1.0, 2.0)}]
    ref = (native.InstanceUpdate * 3)()
    for k, u in enumerate(ups):
        ref[k].instance_index, ref[k].flags = u["instance"], u.get("flags", 0)
        ref[k].translation[:] = u.get("translation", (0.0, 0.0, 0.0))
        ref[k].rotation[:] = u.get("rotation", (0.0, 0.0, 0.0, 1.0))
        ref[k].scale[:] = u.get("scale", (1.0, 1.0, 1.0))
    assert update(ups) == bytes(ref)


@pytest.mark.parametrize("bad", [
    {"translation": (1, 2, 3, 1), "rotation": (0.1, 0.2, 0.3)},
    {"rotation": (0, 0, 0), "scale": (1, 1, 1, 1)},
    {"translation": (1, 2), "scale": np.ones(4)},
    {"translation": (1, 2), "rotation": (0, 0, 0, 1, 1)},
    {"scale": (1, 1)},
    {"translation": {1.0, 2.0, 3.0}},
    {"rotation": iter((0.0, 0.0, 0.0, 1.0))},
    {"scale": "abc"},
])
def test_wrong_shapes_are_refused(bad):
    with pytest.raises((ValueError, TypeError)):
        update([{"instance": 0}, {"instance": 1, **bad}])
