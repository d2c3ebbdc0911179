"""The split plan's pass after each step (CFL of the sides between tiles, the
next step's hanging-edge gradients) against the multi-pass step, bit for bit:
tile sizes, theta, a mesh of one tile (no side between tiles), batches cut short
by their target, a batch without a step, and an all-dry start."""
import numpy as np
import pytest

from test_gpu_resident import FIELDS, gradients, grid, quadtree

pytestmark = pytest.mark.gpu


def dry(w):
    w.initial_depth = np.zeros_like(w.initial_depth)
    return w


CASES = {
    'quadtree': lambda: quadtree(1200),
    'quadtree_theta': lambda: quadtree(1600, theta=0.7),
    'quadtree_dry': lambda: dry(quadtree(1200)),
    'one_tile': lambda: grid(13, 11, horton=True),
    'grid_rows': lambda: grid(61, 47, rows=True),
}


@pytest.mark.parametrize('path', ['tile256', 'tile512', 'tile1024'])
@pytest.mark.parametrize('name', sorted(CASES))
def test_split_step_equals_multipass(cuda_available, name, path):
    from nhflood.native import CudaEngine
    from nhflood.plain import PlainRun
    w = CASES[name]()

    def engine(which):
        def factory(arrays, params):
            params.path, params.cfl = which, 'pass' if which != 'multipass' else 'auto'
            made = CudaEngine(arrays, params)
            assert which == 'multipass' or 'edges=' in made.path, made.path
            return made
        return factory

    a, b = PlainRun(w, engine(path)), PlainRun(w, engine('multipass'))
    for k in range(8):
        if k == 5:   # no step in this batch: the gradients stay the last step's
            now = a.clock.host_now_seconds
            for r in (a, b):
                r.clock.read_trace(r.engine.run_batch(*r.clock.begin(now, now)))
        else:
            ra, rb = (r.engine.run_batch(*r.begin()) for r in (a, b))
            np.testing.assert_array_equal(ra, rb)
            a.finish(ra), b.finish(rb)
        np.testing.assert_array_equal(gradients(a.engine), gradients(b.engine), f'gradients after batch {k}')
    for field in FIELDS:
        np.testing.assert_array_equal(a.engine.get(field).view(np.uint32), b.engine.get(field).view(np.uint32), field)
    assert a.engine.cfl() == b.engine.cfl()
    for x, y in zip(a.engine.limits(), b.engine.limits()):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(a.engine.budget_flush(), b.engine.budget_flush())
    a.close(), b.close()


def test_members_take_the_split_plan(cuda_available):
    """Meshes with hanging edges take the pass at any size (it carries the
    gradients that are a launch of their own otherwise)."""
    from nhflood.native import CudaEngine
    from nhflood.plain import PlainRun
    def factory(arrays, params):
        params.path = 'steps'
        return CudaEngine(arrays, params)
    run = PlainRun(quadtree(1200), factory)
    assert 'cfl=pass' in run.engine.path
    run.close()
    run = PlainRun(grid(40, 40), factory)
    assert 'cfl=fused' in run.engine.path
    run.close()
