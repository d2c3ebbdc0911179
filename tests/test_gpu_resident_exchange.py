"""What the blocks of a resident batch tell one another beyond the state: the
limiting side's snapshot, whose owner changes from step to step; and a batch
whose blocks lose one another (a wait that may not wait runs out)."""
import numpy as np
import pytest

from test_gpu_resident import assert_same, engine, grid, quadtree

pytestmark = pytest.mark.gpu


def torrent(nx=400, ny=24):
    """Reservoirs of growing depth that empty down a slope: the time step's limit
    falls from step to step, and the side that sets it moves from tile to tile."""
    from nhflood import workloads as wl
    from nhflood.forcing import Forcing
    from nhflood.geometry import MeshGeometry
    from nhflood.input import LandParameters
    yy, xx = np.mgrid[:ny, :nx]
    bed = (0.02 * (nx - xx) + 0.05 * yy).astype(np.float32)
    mesh = wl.uniform_grid(nx, ny, 5.0, bed, np.ones((ny, nx), np.uint8), 32)
    geometry = MeshGeometry.from_mesh(mesh)
    rain, _ = wl._uniform_rain(geometry, nx * 5.0, ny * 5.0, np.array([0.]), np.array([900.]), [0.0])
    depth = np.zeros(mesh.e_num, np.float32)
    depth[1:] = np.where(mesh.x[1:] % 320.0 < 100.0, 1.0 + mesh.x[1:] / 500.0, 0.0)
    return wl.Workload('torrent', mesh, geometry, Forcing.assemble([], rain, 900),
                       {1: LandParameters(manning_n=0.012, infiltration='none')}, duration=900, yield_step=300,
                       initial_depth=depth)


@pytest.mark.parametrize('batch', [5, 64])
def test_snapshot_of_changing_owners(cuda_available, batch):
    from nhflood.plain import PlainRun
    w = torrent()
    a, b = (PlainRun(w, engine(path), batch_size=batch) for path in ('auto', 'steps'))
    one = PlainRun(w, engine('steps'), batch_size=1)
    owners = [set()]
    while len(owners) <= 4:
        ra, rb = (r.engine.run_batch(*r.begin()) for r in (a, b))
        np.testing.assert_array_equal(ra, rb)
        a.finish(ra), b.finish(rb)
        while one.elapsed < a.elapsed:
            one.advance()
            owners[-1].add(int(one.engine.limits()[1][1]) // 256)
        assert_same(a, b)
        owners.append(set())
    if batch == 64:
        assert len(owners[0]) > 3    # tiles that held the limit during the first batch
    for r in (a, b, one):
        r.close()


STALLED = 5


@pytest.mark.parametrize('make', [lambda: grid(83, 61), lambda: grid(70, 33, rows=True, theta=0.8), lambda: quadtree(1200)],
                         ids=['grid', 'theta', 'quadtree'])
def test_a_stalled_batch_is_reported_until_initialize(cuda_available, monkeypatch, make):
    import time
    from nhflood.native import CudaEnsemble
    from nhflood.plain import PlainRun
    w = make()
    arrays = w.step_arrays()
    monkeypatch.setenv('NHF_RESIDENT_SPINS', '0')    # read by nhf_initialize
    run = PlainRun(w, engine('auto'), arrays=arrays)
    words = run.begin()
    started = time.perf_counter()
    rows = run.engine.run_batch(*words)
    assert time.perf_counter() - started < 5
    assert rows[0, 3] == STALLED
    with pytest.raises(RuntimeError, match='lost one another'):
        run.finish(rows)
    assert run.clock.pending and run.clock.now_ticks == 0
    # later batches of the handle say the same, resident, as member graphs and in one launch
    assert run.engine.run_batch(*words)[0, 3] == STALLED
    other = PlainRun(w, engine('steps'), arrays=arrays)
    for blocks in (-2, -1):
        ens = CudaEnsemble([run.engine, other.engine], blocks)
        theirs = other.begin()
        traces = ens.run_batch(*(np.array(x, np.uint32) for x in zip(words, theirs)))
        assert traces[0][0, 3] == STALLED and (traces[0][1:, 3] == 0).all()
        other.finish(traces[1])
        ens.close()
    other.close()
    # initialized again with the usual limit: a run like any other
    monkeypatch.delenv('NHF_RESIDENT_SPINS')
    run.engine.budget_flush()
    run.engine.reset_limits()
    for name in ('q', 'rain_time'):
        run.engine.set(name, np.zeros_like(run.engine.get(name)))
    again, fresh = PlainRun(w, lambda a, p: run.engine, arrays=arrays), PlainRun(w, engine('auto'), arrays=arrays)
    for _ in range(3):
        again.advance(), fresh.advance()
    assert again.steps == fresh.steps > 32
    assert_same(again, fresh)
    again.close(), fresh.close()
