"""The CFL candidate where discharges or depths are not numbers: every step form
takes the least of the values that are, with its lowest side, and has none where
there is none (the clock then stops), as the multi-pass step does."""
import dataclasses

import numpy as np
import pytest

from test_gpu_resident import FIELDS, grid

pytestmark = pytest.mark.gpu

FORMS = {'resident': ('auto', 'auto'), 'lattice': ('lattice', 'auto'), 'fused': ('tile256', 'fused'),
         'fused_512': ('tile512', 'fused'), 'split': ('tile256', 'pass')}
NAN, INF = np.float32(np.nan), np.float32(np.inf)


def flat(depth, nx=70, ny=60):
    """A level bed without boundaries or rain."""
    w = grid(nx, ny)
    bed = np.zeros_like(w.mesh.z)
    rain = dataclasses.replace(w.forcing.rain, millimetres=0 * w.forcing.rain.millimetres)
    mesh = dataclasses.replace(w.mesh, z=bed)
    return dataclasses.replace(w, mesh=mesh, forcing=dataclasses.replace(w.forcing, boundaries=[], rain=rain),
                               initial_depth=depth(w.mesh).astype(np.float32))


def cells(mesh):
    return np.concatenate([[0.0], np.ones(mesh.e_num - 1)])


def all_nan():
    w = flat(cells)
    return w, np.full(w.mesh.s_num, NAN, np.float32), None


def lowest_side_nan():
    """Two wet cells with no number on any of their sides, the lowest interior
    side among them, in a dry field."""
    w = flat(lambda m: 0 * cells(m))
    interior = (w.mesh.topology[:, 1] != 0) & (w.mesh.topology[:, 2] != 0)
    pair = w.mesh.topology[np.flatnonzero(interior)[0], 1:]
    depth = np.zeros(w.mesh.e_num, np.float32)
    depth[pair] = 1.0
    q = np.where(np.isin(w.mesh.topology[:, 1:], pair).any(axis=1), NAN, 0).astype(np.float32)
    return dataclasses.replace(w, initial_depth=depth), q, None


def scattered(values):
    def make():
        w = grid(70, 60, horton=True)
        rng = np.random.default_rng(11)
        q = rng.normal(0, 0.3, w.mesh.s_num).astype(np.float32)
        hit = rng.uniform(size=q.size) < 0.02
        q[hit] = rng.choice(np.array(values, np.float32), hit.sum())
        return w, q, None
    return make


def infinite_depths():
    w = grid(70, 60)
    rng = np.random.default_rng(12)
    depth = w.initial_depth.copy()
    depth[1 + rng.choice(w.mesh.e_num - 1, 9, replace=False)] = INF
    return w, None, depth


STATES = {'all_nan': all_nan, 'lowest_side_nan': lowest_side_nan, 'scattered_nan': scattered([NAN]),
          'scattered_infinite': scattered([INF, -INF, NAN]), 'infinite_depths': infinite_depths}


@pytest.mark.parametrize('form', sorted(FORMS))
@pytest.mark.parametrize('state', sorted(STATES))
def test_same_candidate_as_multipass(cuda_available, state, form):
    from nhflood.clock import BAD_CFL
    from nhflood.native import CudaEngine
    from nhflood.plain import PlainRun
    w, q, depth = STATES[state]()

    def engine(path, cfl):
        def factory(arrays, params):
            params.path, params.cfl = path, cfl
            made = CudaEngine(arrays, params)
            assert made.path.startswith({'lattice': 'lattice', 'multipass': 'multipass'}.get(path, 'tiled')), made.path
            assert ('resident' in made.path) == (path == 'auto'), made.path
            return made
        return factory

    runs = [PlainRun(w, engine(*FORMS[form]), batch_size=1), PlainRun(w, engine('multipass', 'auto'), batch_size=1)]
    for r in runs:
        if q is not None:
            q[0] = 0.0     # side 0 stands for none
            r.engine.set('q', q)
        if depth is not None:
            r.engine.set('depth', depth)
    stopped = False
    for step in range(12):
        words = [r.begin() for r in runs]
        a, b = (r.engine.run_batch(*v) for r, v in zip(runs, words))
        np.testing.assert_array_equal(a, b, f'trace of step {step}')
        (ndt, arg), (want, want_arg) = (r.engine.cfl()[:2] for r in runs)
        assert np.float32(ndt).view(np.uint32) == np.float32(want).view(np.uint32) and arg == want_arg, step
        for field in FIELDS:
            have, exact = (r.engine.get(field) for r in runs)
            if field == 'max_speed':     # a speed that is not a number: the multi-pass step keeps it, the others do not
                have, exact = (v[~np.isnan(exact)] for v in (have, exact))
            np.testing.assert_array_equal(have, exact, f'{field} after step {step}')
        if a[0, 3] == BAD_CFL:
            stopped = True
            break
        for r in runs:
            r.finish(a)
    assert stopped == (state in ('all_nan', 'infinite_depths'))    # the latter: a candidate of zero
    for r in runs:
        r.close()
