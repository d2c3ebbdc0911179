"""The lattice march's inner path (warps whose cells are all live and off the
boundaries), its idle rows and its dry CFL key against the tiled step, bit for
bit: grids whose inner warps are none, few and most, cells of 1 m, 4 m and 10 m
(exact inverses or not), dry land with and without rain, an all-dry start, rain
pixels, Horton soil, and extrema below zero."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ('depth', 'q', 'rain_time', 'infiltration', 'max_depth', 'max_speed', 'u', 'v', 'peak_hi', 'peak_lo')


def workload(nx, ny, dx, *, rain=0.0, pixels=1, horton=False, wet='pool', seed=5):
    from nhflood import workloads as wl
    from nhflood.forcing import Forcing, RainField, TimeSeries, select_boundary
    from nhflood.geometry import MeshGeometry
    from nhflood.input import LandParameters
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[:ny, :nx]
    bed = 0.003 * dx * yy + rng.uniform(0, 0.02 * dx, (ny, nx))
    mesh = wl.uniform_grid(nx, ny, dx, bed.astype(np.float32), (1 + (xx // 9) % 2).astype(np.uint8), 32)
    geometry = MeshGeometry.from_mesh(mesh)
    series = TimeSeries(np.array([0., 900.]), np.array([-50., -50.]))
    south = select_boundary('s', 'level', [np.array([[0, 0], [nx * dx, 0]])], series, geometry,
                            np.zeros(mesh.e_num, bool))
    index = np.zeros(mesh.e_num, np.int32)
    index[1:] = ((mesh.x[1:] / dx).astype(np.int32) // 30 + (mesh.y[1:] / dx).astype(np.int32) // 40) % pixels
    rates = rain * rng.uniform(0, 1, (1, pixels)) * (np.arange(pixels) % 3 != 1)     # some pixels without rain
    field = RainField(np.array([0.]), np.array([900.]), rates * 0.25, index)
    soil = dict(f0_mm_h=60.0, fc_mm_h=10.0, k_per_h=4.0) if horton else 'none'
    lands = {1: LandParameters(manning_n=0.03, infiltration='none'), 2: LandParameters(manning_n=0.05, infiltration=soil)}
    depth = np.zeros(mesh.e_num, np.float32)
    if wet == 'pool':
        depth[1:] = np.where((mesh.x[1:] < 0.3 * nx * dx) & (mesh.y[1:] > 0.4 * ny * dx), 0.05 * dx, 0)
    return wl.Workload('grid', mesh, geometry, Forcing.assemble([south], field, 900), lands, duration=900,
                       yield_step=60, initial_depth=depth)


CASES = {
    'no_inner_warp': (dict(nx=57, ny=40, dx=10.0), 4),
    'inner_10m': (dict(nx=150, ny=130, dx=10.0, rain=60.0, pixels=4), 4),
    'inner_1m': (dict(nx=141, ny=97, dx=1.0), 16),
    'inner_4m_horton': (dict(nx=200, ny=160, dx=4.0, rain=90.0, pixels=7, horton=True), 8),
    'all_dry': (dict(nx=113, ny=121, dx=10.0, wet='dry'), 4),
    'dry_then_rain': (dict(nx=113, ny=121, dx=2.0, wet='dry', rain=200.0, pixels=3), 4),
    'tall': (dict(nx=29, ny=900, dx=10.0, rain=40.0, horton=True), 16),
}


@pytest.mark.parametrize('negative', [False, True])
@pytest.mark.parametrize('name', sorted(CASES))
def test_lattice_equals_tiles(cuda_available, monkeypatch, name, negative):
    from nhflood.native import CudaEngine
    from nhflood.plain import PlainRun
    kw, rows = CASES[name]
    monkeypatch.setenv('NHF_LATTICE_ROWS', str(rows))
    w = workload(**kw)

    def engine(path):
        def factory(arrays, params):
            params.path = path
            made = CudaEngine(arrays, params)
            assert made.path.startswith('lattice' if path == 'lattice' else 'tiled'), made.path
            return made
        return factory

    a, b = PlainRun(w, engine('lattice')), PlainRun(w, engine('tiled'))
    if negative:     # extrema a dry cell's zero would raise
        for r in (a, b):
            for field in ('max_depth', 'max_speed'):
                v = r.engine.get(field).copy()
                v[5:4000:7] = -1.0
                r.engine.set(field, v)
    for _ in range(6):
        ra, rb = (r.engine.run_batch(*r.begin()) for r in (a, b))
        np.testing.assert_array_equal(ra, rb)
        a.finish(ra), b.finish(rb)
    for field in FIELDS:
        np.testing.assert_array_equal(a.engine.get(field).view(np.uint32), b.engine.get(field).view(np.uint32), field)
    assert a.engine.cfl() == b.engine.cfl()
    for x, y in zip(a.engine.limits(), b.engine.limits()):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(a.engine.budget_flush(), b.engine.budget_flush())
    a.close(), b.close()
