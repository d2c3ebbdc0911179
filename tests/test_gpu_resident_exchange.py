"""What the blocks of a resident batch tell one another beyond the state: the
limiting side's snapshot, whose owner changes from step to step."""
import numpy as np
import pytest

from test_gpu_resident import assert_same, engine

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
