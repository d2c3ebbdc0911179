"""Handles that take a gate controller after they are made: every choice of step
that leads to 256-cell tiles with a separate CFL pass, or to the multi-pass step,
runs as the gated engine does, bit for bit."""
import numpy as np
import pytest

from test_gpu_resident import FIELDS

pytestmark = pytest.mark.gpu


def attached_later(path, cfl):
    """An engine made without the controller, which is attached then."""
    def factory(arrays, params):
        from nhflood.native import CudaEngine
        tables, arrays.gate = arrays.gate, None
        params.path, params.cfl = path, cfl
        try:
            engine = CudaEngine(arrays, params)
        finally:
            arrays.gate = tables
        engine.gate = tables
        engine._attach_gate(tables)
        return engine
    return factory


@pytest.mark.parametrize('n, path, cfl', [
    (512, 'auto', 'pass'),      # 262,144 cells: the lattice form's size from 2^18 on
    (549, 'auto', 'pass'),      # 301,401: the largest with 256-cell tiles
    (128, 'auto', 'pass'),
    (96, 'multipass', 'auto'),
    (616, 'tile256', 'auto'),   # 1,483 tiles: the pass by size
])
def test_gate_attached_later(cuda_available, n, path, cfl):
    from nhflood.native import CudaEngine
    from nhflood.plain import PlainRun
    from nhflood.workloads import gated_polder
    w = gated_polder(n=n, duration=600)
    runs = [PlainRun(w, f) for f in (attached_later(path, cfl), lambda a, p: CudaEngine(a, p))]
    for _ in range(2):
        a, b = (r.engine.run_batch(*r.begin()) for r in runs)
        np.testing.assert_array_equal(a, b)
        for r in runs:
            r.finish(a)
    for field in FIELDS + ('bed',):
        np.testing.assert_array_equal(*(r.engine.get(field).view(np.uint32) for r in runs), field)
    np.testing.assert_array_equal(*(r.engine.gate_flush() for r in runs))
    for r in runs:
        r.close()


def test_resident_handle_of_an_ensemble_is_refused(cuda_available):
    """A resident handle takes no controller, before and after an ensemble has
    given it a plan of 256-cell tiles with a separate pass."""
    from test_gpu_resident import quadtree
    from nhflood.gate import GateTables
    from nhflood.native import CudaEngine, CudaEnsemble
    from nhflood.plain import PlainRun
    w = quadtree(1200)
    e = w.mesh.e_num
    none = np.zeros(0, np.int32)
    tables = GateTables(1, np.full(e, -1, np.int32), np.zeros(e, np.int32), np.zeros(e, np.float32), none,
                        np.ones(1, np.int32), none, 0, 1.0, 1.0, 0.0)
    run = PlainRun(w, lambda a, p: CudaEngine(a, p))
    assert 'resident=' in run.engine.path
    with pytest.raises(RuntimeError, match='gate control runs'):
        run.engine._attach_gate(tables)
    ens = CudaEnsemble([run.engine], -2)
    with pytest.raises(RuntimeError, match='gate control runs'):
        run.engine._attach_gate(tables)
    ens.close()
    run.close()
