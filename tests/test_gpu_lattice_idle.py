"""Rows that the lattice march may not take for idle although they are dry and no
water moves: a wet threshold of zero (dry cells count as wet), infiltration below
zero or not a number, rain below zero. Against the tiled step, bit for bit."""
import dataclasses

import numpy as np
import pytest

from test_gpu_lattice import FIELDS, workload

pytestmark = pytest.mark.gpu


def infiltration(value):
    def change(run):
        v = run.engine.get('infiltration').copy()
        v[3000:9000:11] = value
        run.engine.set('infiltration', v)
    return change


CASES = {
    'threshold_zero': (dict(), dict(min_h=0.0), None),
    'infiltration_negative': (dict(), dict(), infiltration(-2e-5)),
    'infiltration_nan': (dict(), dict(), infiltration(np.nan)),
    'rain_negative': (dict(rain=-60.0, pixels=4), dict(), None),
}


@pytest.mark.parametrize('name', sorted(CASES))
def test_lattice_equals_tiles(cuda_available, monkeypatch, name):
    from nhflood.native import CudaEngine
    from nhflood.plain import PlainRun
    kw, fields, change = CASES[name]
    monkeypatch.setenv('NHF_LATTICE_ROWS', '4')
    w = dataclasses.replace(workload(150, 130, 10.0, **kw), **fields)

    def engine(path):
        def factory(arrays, params):
            params.path = path
            made = CudaEngine(arrays, params)
            assert made.path.startswith(path), made.path
            return made
        return factory

    a, b = PlainRun(w, engine('lattice')), PlainRun(w, engine('tiled'))
    if change is not None:
        for r in (a, b):
            change(r)
    for _ in range(3):
        ra, rb = (r.engine.run_batch(*r.begin()) for r in (a, b))
        np.testing.assert_array_equal(ra, rb)
        a.finish(ra), b.finish(rb)
    for field in FIELDS:
        np.testing.assert_array_equal(a.engine.get(field).view(np.uint32), b.engine.get(field).view(np.uint32), field)
    np.testing.assert_array_equal(a.engine.budget_flush(), b.engine.budget_flush())
    a.close(), b.close()
