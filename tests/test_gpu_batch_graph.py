"""A batch's captured graph and the buffers it holds the addresses of: a run that
makes one of them grow must not leave a graph that writes to the old one."""
import numpy as np
import pytest

from tests.test_gpu_batch import bits, films, small_jobs
from vkpathtracer_b200.tracer import BatchRenderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("between", [
    dict(mode="loop", use_graph=False, stack_depth=1),                    # the stack spill
    dict(mode="persistent", use_graph=False, stack_depth=1),
    dict(mode="loop", use_graph=False, stack_depth=8, pool_paths=1 << 17),   # the pool
    dict(mode="persistent", use_graph=False, stack_depth=8, pool_paths=1 << 17),
    dict(mode="loop", stack_depth=8, sample_limit=0),                     # the staging
])
@pytest.mark.parametrize("mode", ["loop", "persistent"])
def test_graph_follows_its_buffers(mode, between):
    n = len(small_jobs())
    first = dict(mode=mode, stack_depth=8, pool_paths=1 << 14, sample_limit=2)
    with BatchRenderer() as b:
        for sc, st in small_jobs():
            b.add_job(sc, st)
        b.run("plain", sample_limit=2)
        plain = films(b, n)
        for kw in (first, between, first, first):
            stats = b.run(**kw)
        assert stats["graph_used"] == 1
        for (f, c), (pf, pc) in zip(films(b, n), plain):
            assert np.array_equal(c, pc) and np.array_equal(bits(f), bits(pf))
