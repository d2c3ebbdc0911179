"""Handles whose own batches run in another form than tiles, in a one-launch
ensemble: each member as alone, bit for bit."""
import numpy as np
import pytest

from test_gpu_resident import assert_same, grid, quadtree

pytestmark = pytest.mark.gpu


def auto(arrays, params):
    from nhflood.native import CudaEngine
    return CudaEngine(arrays, params)


@pytest.mark.parametrize('blocks', [0, -1])
@pytest.mark.parametrize('form, works', [
    ('lattice', [lambda: grid(520, 592, horton=True), lambda: grid(640, 500)]),    # the lattice's sizes from 2^18 cells on
    ('resident', [lambda: grid(60, 47), lambda: quadtree(1200)]),
])
def test_one_launch(cuda_available, form, works, blocks):
    from nhflood.native import CudaEnsemble
    from nhflood.plain import PlainRun
    works = [w() for w in works]
    together, alone = ([PlainRun(w, auto) for w in works] for _ in range(2))
    assert all(form in r.engine.path for r in together)
    ens = CudaEnsemble([r.engine for r in together], blocks)
    for _ in range(2):
        words = [r.begin() for r in together]
        traces = ens.run_batch(*(np.array(x, np.uint32) for x in zip(*words)))
        for a, b, rows in zip(together, alone, traces):
            want = b.engine.run_batch(*b.begin())
            np.testing.assert_array_equal(rows, want)
            a.finish(rows), b.finish(want)
        for a, b in zip(together, alone):    # a member's own batch between the ensemble's
            a.advance(), b.advance()
            assert_same(a, b)
    ens.close()
    for r in together + alone:
        r.close()


def test_a_requested_lattice_is_refused(cuda_available):
    from nhflood.native import CudaEngine, CudaEnsemble
    from nhflood.plain import PlainRun

    def lattice(arrays, params):
        params.path = 'lattice'
        return CudaEngine(arrays, params)
    run = PlainRun(grid(70, 60), lattice)
    assert run.engine.path.startswith('lattice')
    with pytest.raises(RuntimeError, match='not on the fused tiled step'):
        CudaEnsemble([run.engine], -1)
    run.close()
