"""A handle initialized a second time after its caller changed the side lengths:
nothing laid out by the first call stays in use."""
import numpy as np
import pytest

from test_gpu_cfl_not_a_number import cells, flat
from test_gpu_resident import FIELDS, quadtree

pytestmark = pytest.mark.gpu


def run_with(path, make, factor):
    """A run whose side lengths, and face sums with them, are scaled after a
    first initialize; None for one made with them."""
    from nhflood.native import CudaEngine
    from nhflood.plain import PlainRun
    w = make()
    arrays = w.step_arrays()
    if factor is None:
        arrays.length = arrays.length * np.float32(2)

    def factory(a, params):
        params.path = path
        engine = CudaEngine(a, params)
        if factor is not None:
            engine.initialize()
            engine.t['length'].mul_(factor)
        return engine
    return PlainRun(w, factory, arrays=arrays)


@pytest.mark.parametrize('path', ['auto', 'steps', 'tile512', 'multipass'])
@pytest.mark.parametrize('make', [lambda: flat(lambda m: 0 * cells(m)), lambda: quadtree(1200)], ids=['dry', 'quadtree'])
def test_second_initialize(cuda_available, path, make):
    again, fresh = run_with(path, make, 2.0), run_with(path, make, None)
    for _ in range(3):
        a, b = (r.engine.run_batch(*r.begin()) for r in (again, fresh))
        np.testing.assert_array_equal(a, b)
        again.finish(a), fresh.finish(b)
    assert again.engine.cfl() == fresh.engine.cfl()
    for field in FIELDS:
        np.testing.assert_array_equal(*(r.engine.get(field).view(np.uint32) for r in (again, fresh)), field)
    for r in (again, fresh):
        r.close()
