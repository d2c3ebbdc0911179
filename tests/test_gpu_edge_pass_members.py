"""The split plan's pass after each step where its gradient blocks may start
late, after other blocks of the pass have finished: many quadtree members
sharing the GPU in the member graphs, and one mesh whose pass is more blocks than
the GPU holds at once. Traces, gradients and state against the multi-pass step,
bit for bit, after every batch."""
import numpy as np
import pytest

from test_gpu_resident import FIELDS, gradients, quadtree

pytestmark = pytest.mark.gpu


def engine(path):
    def factory(arrays, params):
        from nhflood.native import CudaEngine
        params.path = path
        made = CudaEngine(arrays, params)
        assert ('edges=' in made.path) == (path == 'steps'), made.path
        return made
    return factory


def assert_same(a, b, where):
    np.testing.assert_array_equal(gradients(a.engine), gradients(b.engine), f'gradients, {where}')
    for field in FIELDS:
        np.testing.assert_array_equal(a.engine.get(field).view(np.uint32), b.engine.get(field).view(np.uint32),
                                      f'{field}, {where}')


def test_members_together(cuda_available):
    from nhflood.native import CudaEnsemble
    from nhflood.plain import PlainRun
    works = [quadtree(1200 + 400 * (i % 5), theta=0.7 if i % 4 == 3 else 1.0) for i in range(12)]
    together = [PlainRun(w, engine('steps')) for w in works]
    alone = [PlainRun(w, engine('multipass')) for w in works]
    ens = CudaEnsemble([r.engine for r in together], -2)
    for batch in range(8):
        targets, origins = (np.array(x, np.uint32) for x in zip(*(r.begin() for r in together)))
        traces = ens.run_batch(targets, origins)
        for i, (a, b) in enumerate(zip(together, alone)):
            rows = b.engine.run_batch(*b.begin())
            np.testing.assert_array_equal(traces[i], rows)
            a.finish(traces[i]), b.finish(rows)
            assert_same(a, b, f'member {i}, batch {batch}')
    ens.close()
    for r in together + alone:
        r.close()


def test_pass_of_more_than_a_wave(cuda_available):
    """The pass has more blocks than the five per SM that its registers allow."""
    import torch
    from nhflood.plain import PlainRun
    w = quadtree(20000)
    arrays = w.step_arrays()
    a, b = (PlainRun(w, engine(path), arrays=arrays) for path in ('steps', 'multipass'))
    edges = int(a.engine.path.split('edges=')[1].rstrip(')'))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert edges // 256 + 2 * arrays.hang_cells // 256 > 5 * sms
    for batch in range(3):
        ra, rb = (r.engine.run_batch(*r.begin()) for r in (a, b))
        np.testing.assert_array_equal(ra, rb)
        a.finish(ra), b.finish(rb)
        assert_same(a, b, f'batch {batch}')
    a.close(), b.close()
