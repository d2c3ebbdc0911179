"""The resident form (a batch in one cooperative launch) against the step by
step form, bit for bit: traces, state, extrema, budget, limiting side,
gradients and clock, at the edges of its tiles (one cell short of a tile, one
more; one block, all blocks), over both numberings, hanging edges, theta < 1,
level and discharge boundaries, Horton soil, batches cut short by their target
and batches of one and of 64 steps."""
import ctypes
import dataclasses
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ('depth', 'q', 'rain_time', 'infiltration', 'max_depth', 'max_speed', 'u', 'v', 'peak_hi', 'peak_lo')


def engine(path):
    def factory(arrays, params):
        from nhflood.native import CudaEngine
        params.path = path
        made = CudaEngine(arrays, params)
        assert ('resident=' in made.path) == (path == 'auto'), made.path
        return made
    return factory


def grid(nx, ny, *, rows=False, theta=1.0, horton=False, seed=3):
    """A wet hilly grid with a level boundary in the south and a discharge
    boundary (inflow, then extraction) in the north."""
    from nhflood import workloads as wl
    from nhflood.forcing import Forcing, TimeSeries, select_boundary
    from nhflood.geometry import MeshGeometry
    from nhflood.input import LandParameters
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[:ny, :nx]
    bed = 0.02 * yy + rng.uniform(0, 0.3, (ny, nx))
    land = (1 + (xx // 5 + yy // 7) % 2).astype(np.uint8)
    mesh = wl.uniform_grid(nx, ny, 10.0, bed.astype(np.float32), land, max(nx, ny) if rows else 32)
    geometry = MeshGeometry.from_mesh(mesh)
    w, h = nx * 10.0, ny * 10.0
    claimed = np.zeros(mesh.e_num, bool)
    t = np.array([0.0, 40.0, 600.0])
    south = select_boundary('s', 'level', [np.array([[0, 0], [w, 0]])], TimeSeries(t, np.array([0.4, 0.6, 0.5])),
                            geometry, claimed)
    north = select_boundary('n', 'discharge', [np.array([[0, h], [w, h]])],
                            TimeSeries(t, np.array([8.0, -6.0, 4.0])), geometry, claimed)
    rain, _ = wl._uniform_rain(geometry, w, h, np.array([0., 50.]), np.array([50., 600.]), [2.0, 9.0])
    soil = dict(f0_mm_h=60.0, fc_mm_h=10.0, k_per_h=4.0) if horton else 'none'
    lands = {1: LandParameters(manning_n=0.03, infiltration='none'), 2: LandParameters(manning_n=0.06, infiltration=soil)}
    depth = np.zeros(mesh.e_num, np.float32)
    depth[1:] = np.maximum(rng.uniform(-0.1, 0.4, nx * ny), 0)
    return wl.Workload('grid', mesh, geometry, Forcing.assemble([south, north], rain, 600), lands, duration=600,
                       yield_step=30, sita=theta, initial_depth=depth)


def quadtree(width, theta=1.0):
    from nhflood.workloads import multires_quadtree
    w = multires_quadtree(width=float(width), duration=600)
    depth = np.where(w.mesh.land_type == 0, 1.5, 0.3).astype(np.float32)
    depth[0] = 0.0
    return dataclasses.replace(w, initial_depth=depth, sita=theta, yield_step=20)


CASES = {
    'one_cell_short': (lambda: grid(17, 15), 32, 8),        # 255 cells and the sentinel: one full tile
    'one_cell_more': (lambda: grid(16, 16), 32, 8),         # 256 cells: a second tile of one cell
    'rows': (lambda: grid(131, 61, rows=True, horton=True), 32, 8),
    'theta_rows': (lambda: grid(70, 33, rows=True, theta=0.8), 32, 8),
    'theta_horton': (lambda: grid(90, 50, theta=0.7, horton=True), 7, 20),
    'single_steps': (lambda: grid(40, 33, horton=True), 1, 60),
    'long_batches': (lambda: grid(40, 33), 64, 6),
    'all_blocks': (lambda: grid(148, 256), 32, 3),          # 148 tiles of 256 cells but for the sentinel: 512-cell tiles
    'last_256': (lambda: grid(148, 255), 32, 3),            # 148 tiles of 256 cells
    'tiles_768': (lambda: grid(330, 331), 32, 2),
    'tiles_1024': (lambda: grid(380, 380, horton=True), 32, 2),
    'tiles_1536': (lambda: grid(440, 460), 32, 2),
    'tiles_2048': (lambda: grid(512, 576, horton=True), 32, 2),   # whole 32 x 32 tiles: the halo fits
    'quadtree': (lambda: quadtree(1200), 32, 12),
    'quadtree_theta': (lambda: quadtree(2000, theta=0.7), 32, 6),
    'quadtree_large': (lambda: quadtree(5000), 32, 2),
}


def gradients(e):
    import torch
    out = torch.zeros(2 * max(1, e.arrays.hang_cells), device=e.device)
    e._check(e.lib.nhf_read_gradients(e.h, ctypes.c_void_p(out.data_ptr())), 'nhf_read_gradients')
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint32)


def assert_same(a, b):
    for name in FIELDS:
        np.testing.assert_array_equal(a.engine.get(name).view(np.uint32), b.engine.get(name).view(np.uint32), name)
    np.testing.assert_array_equal(a.engine.get_clock(), b.engine.get_clock())
    assert a.engine.cfl() == b.engine.cfl()
    for x, y in zip(a.engine.limits(), b.engine.limits()):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(gradients(a.engine), gradients(b.engine))
    np.testing.assert_array_equal(a.engine.budget_flush(), b.engine.budget_flush())


@pytest.mark.parametrize('name', sorted(CASES))
def test_resident_equals_step_by_step(cuda_available, name):
    from nhflood.plain import PlainRun
    make, batch, batches = CASES[name]
    w = make()
    arrays = w.step_arrays()
    a, b = (PlainRun(w, engine(path), batch_size=batch, arrays=arrays) for path in ('auto', 'steps'))
    cut = 0
    for k in range(batches):
        ra, rb = (r.engine.run_batch(*r.begin()) for r in (a, b))
        np.testing.assert_array_equal(ra, rb)
        cut += int((ra[:, 3] != 1).any())
        a.finish(ra)
        b.finish(rb)
        if k == batches // 2:
            assert_same(a, b)
    # a batch whose target is the clock: no step, the state as it is
    now = a.clock.host_now_seconds
    for r in (a, b):
        rows = r.engine.run_batch(*r.clock.begin(now, now))
        assert (rows[:, 3] == 0).all()
        r.clock.read_trace(rows)
    a.advance(), b.advance()
    assert_same(a, b)
    if name in ('one_cell_more', 'long_batches', 'quadtree'):
        assert cut > 0      # some batch was cut short by its target
    a.close()
    b.close()


def test_tile_choice(cuda_available):
    """One tile per SM at most; the next size from the first cell that does
    not fit (148 SMs)."""
    from nhflood.plain import PlainRun
    for cells, tile in ((148 * 255, 256), (148 * 256, 512)):
        run = PlainRun(grid(148, cells // 148), engine('auto'))
        assert run.engine.path.startswith(f'tiled(tile={tile},'), run.engine.path
        run.close()


def test_resident_runs_on_two_threads(cuda_available):
    """Two solves in two threads on their own streams: each as alone."""
    import torch
    from nhflood.plain import PlainRun
    works = [grid(200, 190, horton=True), quadtree(2400)]
    alone = []
    for w in works:
        run = PlainRun(w, engine('auto'))
        for _ in range(6):
            run.advance()
        alone.append({k: run.engine.get(k) for k in FIELDS})
        run.close()
    got = [None, None]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            run = PlainRun(works[i], engine('auto'))
            for _ in range(6):
                run.advance()
            got[i] = {k: run.engine.get(k) for k in FIELDS}
            run.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for want, have in zip(alone, got):
        for k in FIELDS:
            np.testing.assert_array_equal(want[k].view(np.uint32), have[k].view(np.uint32), k)


def test_resident_handle_in_an_ensemble(cuda_available):
    """A handle made for resident batches joins the member graphs (its step
    plan is made then) and goes on resident afterwards."""
    from nhflood.native import CudaEnsemble
    from nhflood.plain import PlainRun
    works = [grid(60, 47), quadtree(1200)]
    mixed, plain = ([PlainRun(w, engine(path)) for w in works] for path in ('auto', 'steps'))
    ens = CudaEnsemble([r.engine for r in mixed], -2)
    for k in range(3):
        words = [r.begin() for r in mixed]
        traces = ens.run_batch(*(np.array(x, np.uint32) for x in zip(*words)))
        for r, t in zip(mixed, traces):
            r.finish(t)
        for r in mixed:
            r.advance()
        for r in plain:
            r.advance()
            r.advance()
    for a, b in zip(mixed, plain):
        assert_same(a, b)
    ens.close()
