"""The work this framework is used for, as cases that can be timed.

One pass of a case is one device batch (32 time steps) through the calls a
program makes: ``PlainRun.advance`` for one domain (forcing for the batch,
``CudaEngine.run_batch``, the trace), ``EnsembleRun.advance`` for several
domains together. The simulated time goes on from pass to pass under steady
rain, so a case settles into the state a long storm has.

A case names the mesh (kind, size, numbering) and the options (rain raster,
soil, theta); a seed gives the terrain, the water it starts with, the rain and
the tide. Connectivity and land classes belong to the mesh of a case.
"""
from __future__ import annotations

import dataclasses
import math
import sys
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / 'nh-flood-2d_b200'))

from nhflood import workloads as wl  # noqa: E402
from nhflood.ensemble import EnsembleRun  # noqa: E402
from nhflood.forcing import Forcing, RainField, TimeSeries, select_boundary  # noqa: E402
from nhflood.geometry import MeshGeometry  # noqa: E402
from nhflood.input import LandParameters  # noqa: E402
from nhflood.native import CudaEngine  # noqa: E402
from nhflood.plain import PlainRun  # noqa: E402

BATCH = 32
DURATION = 4_000_000        # simulated seconds: no pass reaches the end
STATE = ('depth', 'q', 'rain_time', 'infiltration', 'max_depth', 'max_speed', 'u', 'v')
G = float(np.float32(9.81))
HORTON = dict(f0_mm_h=60.0, fc_mm_h=10.0, k_per_h=4.0)


def listed():
    return [
        # A study of one street block or a teaching case: a few thousand cells,
        # where a step is latency. Numbered row by row, as raster exporters do.
        dict(name='grid_83x61_rows', kind='grid', nx=83, ny=61, order='rows', raster=1, soil='none', theta=1.0),
        # The plain configuration of the benchmark: 256 x 256 cells, two land
        # classes, uniform rain, free outflow in the south.
        dict(name='grid_256x256', kind='grid', nx=256, ny=256, order='tiles', raster=1, soil='none', theta=1.0),
        # A catchment exported from a DEM raster, row by row, with rain radar
        # pixels and Horton soil.
        dict(name='grid_421x307_rows_horton', kind='grid', nx=421, ny=307, order='rows', raster=12, soil='horton',
             theta=1.0),
        # A city district: under a million cells, rain radar, Horton soil.
        dict(name='grid_1003x741_horton', kind='grid', nx=1003, ny=741, order='tiles', raster=20, soil='horton',
             theta=1.0),
        # A whole city at a few metres: millions of cells, storm and soil.
        dict(name='grid_2048x1531_horton', kind='grid', nx=2048, ny=1531, order='tiles', raster=32, soil='horton',
             theta=1.0),
        # The dam break configuration: 16.8 M cells at 1 m, mostly dry land
        # ahead of the wave.
        dict(name='dambreak_4096', kind='dambreak', nx=4096, ny=4096),
        # A small served request: a 2:1 quadtree of some 20,000 cells.
        dict(name='quadtree_1200m', kind='quadtree', width=1200, mesh_seed=11, raster=1, theta=1.0),
        # A median member of the batched and served forms.
        dict(name='quadtree_6km', kind='quadtree', width=6000, mesh_seed=7, raster=1, theta=1.0),
        # The multi-resolution configuration: 20 km x 20 km, 1.36 M cells,
        # storm raster, Horton soil, tide.
        dict(name='quadtree_20km', kind='quadtree', width=20000, mesh_seed=2, raster=100, theta=1.0),
        # The theta-weighted scheme (theta < 1), used where theta = 1 rings.
        dict(name='quadtree_4km_theta', kind='quadtree', width=4000, mesh_seed=5, raster=10, theta=0.7),
        # Gates that open into a polder (the gate controller in every step).
        dict(name='polder_512', kind='polder', nx=512),
        # The batched form: scenarios of uneven size advanced together.
        dict(name='ensemble_6', kind='ensemble', members=6, low=40000, high=400000, mesh_seed=4),
    ]


def draw(rng):
    def log(low, high):
        return math.exp(rng.uniform(math.log(low), math.log(high)))

    kind = rng.choice(['grid', 'grid', 'grid', 'dambreak', 'quadtree', 'quadtree', 'quadtree', 'polder', 'ensemble'])
    if kind == 'grid':
        cells, aspect = log(3e3, 4e6), rng.uniform(0.5, 2.0)
        nx = max(20, round(math.sqrt(cells * aspect)))
        return dict(kind=kind, nx=nx, ny=max(20, round(cells / nx)), order=rng.choice(['tiles', 'tiles', 'rows']),
                    raster=rng.choice([1, 1, rng.randint(2, 40)]), soil=rng.choice(['none', 'horton']),
                    theta=rng.choice([1.0, 1.0, 1.0, round(rng.uniform(0.6, 0.95), 2)]))
    if kind == 'dambreak':
        return dict(kind=kind, nx=round(log(150, 2600)), ny=round(log(150, 2600)))
    if kind == 'quadtree':
        return dict(kind=kind, width=20 * round(log(800, 16000) / 20), mesh_seed=rng.randint(20, 10000),
                    raster=rng.choice([1, rng.randint(2, 60)]),
                    theta=rng.choice([1.0, 1.0, 1.0, round(rng.uniform(0.6, 0.95), 2)]))
    if kind == 'polder':
        return dict(kind=kind, nx=16 * round(log(160, 800) / 16))
    low = log(2e4, 8e4)
    return dict(kind=kind, members=rng.randint(3, 6), low=round(low), high=round(low * rng.uniform(2, 6)),
                mesh_seed=rng.randint(20, 10000))


# ------------------------------------------------------------------- meshes

def _land(manning, horton):
    return {k: LandParameters(manning_n=n, infiltration=HORTON if k and horton else 'none')
            for k, n in enumerate(manning)}


@lru_cache(maxsize=2)
def _grid(nx, ny, dx, tile, horton, line):
    """Mesh, geometry, open cells and step arrays of a uniform grid with flat
    bed; ``line`` is the open edge, 'south' or the whole 'perimeter'."""
    yy, xx = np.divmod(np.arange(nx * ny), nx)
    land = (1 + ((xx // 37 + yy // 53) % 2)).astype(np.uint8)
    mesh = wl.uniform_grid(nx, ny, dx, np.zeros(nx * ny, np.float32), land, tile)
    geometry = MeshGeometry.from_mesh(mesh)
    w, h = nx * dx, ny * dx
    corners = np.array([[0., 0.], [w, 0.]] + ([[w, h], [0., h], [0., 0.]] if line == 'perimeter' else []))
    series = TimeSeries(np.array([0., DURATION]), np.zeros(2))
    boundary = select_boundary(line, 'level', [corners], series, geometry, np.zeros(mesh.e_num, bool))
    return _with_arrays(mesh, geometry, boundary, _land([0.03, 0.03, 0.06], horton))


def _meander(width, mesh_seed):
    return wl.meander_leaves(mesh_seed, float(width), 20.0, buffer=500.0, half_channel=15.0)


@lru_cache(maxsize=64)
def _leaves(width, mesh_seed):
    return len(_meander(width, mesh_seed)[0])


@lru_cache(maxsize=8)
def _quadtree(width, mesh_seed):
    """The repository's meander quadtree (20/10/5 m) with flat bed."""
    lv, li, lj, distance, n0 = _meander(width, mesh_seed)

    def land_at(x, y, level):
        return np.where(distance(x, y) < 15.0, 0, 1 + (x // 370 + y // 530).astype(np.int64) % 3).astype(np.uint8)

    mesh = wl.quadtree_mesh(lv, li, lj, 20.0, 3, n0, n0, lambda x, y, level: np.zeros(len(x), np.float32), land_at)
    geometry = MeshGeometry.from_mesh(mesh)
    line = np.array([[width, 0.], [width, width]], float)
    series = TimeSeries(np.array([0., DURATION]), np.zeros(2))
    boundary = select_boundary('tide', 'level', [line], series, geometry, np.zeros(mesh.e_num, bool))
    return _with_arrays(mesh, geometry, boundary, _land([0.015, 0.035, 0.05, 0.08], True))


def _with_arrays(mesh, geometry, boundary, land):
    rain = RainField(np.array([0.]), np.array([float(DURATION)]), np.zeros((1, 1)), np.zeros(mesh.e_num, np.int32))
    w = wl.Workload('case', mesh, geometry, Forcing.assemble([boundary], rain, DURATION), land, duration=DURATION,
                    yield_step=3600)
    return w, {1.0: w.step_arrays()}


# ------------------------------------------------------------------- inputs

def _device():
    return 'cuda' if torch.cuda.is_available() else 'cpu'


def _noise(gen, ny, nx, octaves=5, base=4):
    """Fractal noise in [0, 1]: random lattices, amplitude halving per octave."""
    out = torch.zeros(ny, nx, device=gen.device)
    for o in range(octaves):
        k = base * 2 ** o + 1
        lattice = torch.rand(1, 1, k, k, generator=gen, device=gen.device)
        out += 0.5 ** o * torch.nn.functional.interpolate(lattice, size=(ny, nx), mode='bilinear',
                                                          align_corners=True)[0, 0]
    out -= out.min()
    return out / out.max()


def _sample(field, x, y, w, h):
    ny, nx = field.shape
    i = (x / w * nx).long().clamp(0, nx - 1)
    j = (y / h * ny).long().clamp(0, ny - 1)
    return field[j, i]


def _numpy(values, e_num):
    out = np.zeros(e_num, np.float32)
    out[1:] = values.float().cpu().numpy()
    return out


def _workload(case, seed):
    """(workload, step arrays) of a case, its values from the seed."""
    if case['kind'] == 'polder':
        w = wl.gated_polder(n=case['nx'], seed=seed, duration=DURATION)
        return w, w.step_arrays()
    gen = torch.Generator(device=_device()).manual_seed(seed)
    host = np.random.default_rng(seed)
    theta = case.get('theta', 1.0)
    quadtree = case['kind'] == 'quadtree'
    if quadtree:
        width = height = float(case['width'])
        base, arrays = _quadtree(case['width'], case['mesh_seed'])
        detail = (512, 512)
    else:
        dambreak = case['kind'] == 'dambreak'
        dx = 1.0 if dambreak else 10.0
        width, height = case['nx'] * dx, case['ny'] * dx
        tile = max(case['nx'], case['ny']) if case.get('order') == 'rows' else 32
        base, arrays = _grid(case['nx'], case['ny'], dx, tile, case.get('soil') == 'horton',
                             'perimeter' if dambreak else 'south')
        detail = (case['ny'], case['nx'])
    if theta not in arrays:
        base.sita = theta
        arrays[theta] = base.step_arrays()
    mesh, e = base.mesh, base.mesh.e_num
    x = torch.from_numpy(mesh.x[1:]).to(gen.device)
    y = torch.from_numpy(mesh.y[1:]).to(gen.device)
    relief = _sample(_noise(gen, *detail), x, y, width, height)
    film = (0.12 * _sample(_noise(gen, *detail), x, y, width, height) - 0.03).clamp(min=0)
    cells = base.forcing.boundaries[0].cells
    if quadtree:       # rolling land draining to a channel and a tidal edge
        channel = torch.from_numpy(mesh.land_type[1:] == 0).to(gen.device)
        bed = _numpy(20.0 * relief + 0.0005 * (width - x) - 3.0 * channel, e)
        depth = _numpy(film + 1.5 * channel, e)
        mean = float(np.percentile(bed[cells], 10)) + 1.0
        level = [mean, mean + host.uniform(0.0, 1.0)]
    elif case['kind'] == 'dambreak':
        bed = _numpy(10.0 * relief + 0.002 * (width - x), e)
        depth = _numpy(2.0 * (x < width * host.uniform(0.2, 0.3)), e)
        level = [float(bed.min()) - 100.0] * 2
    else:              # a slope to the south with hills
        bed = _numpy(0.001 * y + 2.0 * relief, e)
        depth = _numpy(film, e)
        level = [float(bed.min()) - 100.0] * 2
    if case['kind'] == 'dambreak':
        rate, pixels = np.zeros(1), np.zeros(e, np.int32)
    else:
        n = case['raster']
        rate = host.uniform(20.0, 60.0) * (host.uniform(0.0, 1.0, n * n) if n > 1 else np.ones(1))   # mm/h
        pixels = np.zeros(e, np.int32)
        pixels[1:] = (np.minimum(mesh.y[1:] * n / height, n - 1).astype(np.int32) * n
                      + np.minimum(mesh.x[1:] * n / width, n - 1).astype(np.int32))
    rain = RainField(np.array([0.]), np.array([float(DURATION)]), rate[None] * DURATION / 3600.0, pixels)
    boundary = dataclasses.replace(base.forcing.boundaries[0],
                                   series=TimeSeries(np.array([0., DURATION]), np.array(level, float)))
    w = dataclasses.replace(base, mesh=dataclasses.replace(mesh, z=bed), sita=theta, initial_depth=depth,
                            forcing=Forcing.assemble([boundary], rain, DURATION))
    return w, dataclasses.replace(arrays[theta], bed=bed, rain_index=pixels, n_rates=len(rate))


def _members(case):
    rng = np.random.default_rng(case['mesh_seed'])
    for i in range(case['members']):
        cells = math.exp(rng.uniform(math.log(case['low']), math.log(case['high'])))
        yield dict(kind='quadtree', width=20 * max(8, round(wl.quadtree_width_for(cells) / 20)),
                   mesh_seed=1000 * case['mesh_seed'] + i, raster=1, theta=1.0)


def prepare(case, seed):
    if case['kind'] == 'ensemble':
        workloads = []
        for i, m in enumerate(_members(case)):
            w, arrays = _workload(m, seed + 7919 * i)
            w.step_arrays = lambda arrays=arrays: arrays   # already built
            workloads.append(w)
        return EnsembleRun(workloads, batch_size=BATCH)
    w, arrays = _workload(case, seed)
    return PlainRun(w, lambda a, p: CudaEngine(a, p), batch_size=BATCH, arrays=arrays)


def _outputs(run):
    t = run.engine.t
    out = {name: t[name] for name in STATE}
    out['peak_ticks'] = [t['peak_hi'], t['peak_lo']]
    out['steps'], out['elapsed'] = run.steps, run.elapsed
    if run.engine.gate is not None:
        out['bed'] = t['bed']
    return out


def run(state):
    state.advance()
    if isinstance(state, EnsembleRun):
        # at most 64 outputs: the fields a scenario's frames and checkpoints hold
        return [{k: v for k, v in _outputs(r).items() if k in ('depth', 'q', 'infiltration', 'max_depth', 'max_speed',
                                                               'steps', 'elapsed')} for r in state.runs]
    return _outputs(state)


# --------------------------------------------------------------------- work

def work(case):
    """Bytes a step has to move per cell, times the cells and the steps of a
    batch (each step needs the whole state of the one before it): depth, q of
    two sides, max_depth and max_speed read and written, bed and two Manning n
    read; with rain the pixel, with Horton soil rain time and capacity read
    and written and three parameters read; on quadtrees the connectivity."""
    if case['kind'] == 'ensemble':
        parts = [work(m) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ('bytes', 'flops')}
    if case['kind'] == 'quadtree':
        cells = _leaves(case['width'], case['mesh_seed'])
        per = 84 + 44
    else:
        cells = case['nx'] * case.get('ny', case['nx'])
        per = {'dambreak': 52, 'polder': 64}.get(case['kind']) or (84 if case['soil'] == 'horton' else 56)
    return {'bytes': per * cells * BATCH, 'flops': 150 * cells * BATCH}


# -------------------------------------------------- the same batch in 64 bits

def exact(case, seed):
    if case['kind'] == 'polder':
        return None   # beds in motion: the controller's clock decides them
    if case['kind'] == 'ensemble':
        keep = ('depth', 'q', 'infiltration', 'max_depth', 'max_speed', 'steps', 'elapsed')
        parts = [_batch64(*_workload(m, seed + 7919 * i)) for i, m in enumerate(_members(case))]
        return [{k: p[k] for k in keep} for p in parts]
    return _batch64(*_workload(case, seed))


def _batch64(w, a):
    """The first batch of a workload: the local-inertial step in 64 bits."""
    dev = _device()

    def put(v):
        v = torch.from_numpy(np.ascontiguousarray(v)).to(dev)
        return v.double() if v.is_floating_point() else v.long()

    e, min_h, dh = a.e_num, float(np.float32(w.min_h)), -999.0
    orient, lo, hi = put(a.topology).unbind(1)
    vertical = orient == 2
    length, n = put(a.length), put(a.side_n)
    area, width, height = put(a.area), put(a.width), put(a.height)
    bed, x, y = put(a.bed), put(a.x), put(a.y)
    f0, fc, k = put(a.f0), put(a.fc), put(a.k)
    rate = put(w.forcing.rain.rates(0).astype(np.float32))[put(a.rain_index)]
    rate[0] = 0
    level_cell = put(a.boundary_id) >= 0
    series = w.forcing.boundaries[0].series
    start, slope = (float(np.float32(v)) for v in (series.values[0], (series.values[1] - series.values[0])
                                                   / (series.times[1] - series.times[0])))
    dx = torch.where(vertical, (x[hi] - x[lo]).abs(), (y[hi] - y[lo]).abs()).clamp(min=0.01)
    closed = (lo == 0) != (hi == 0)
    inner = (lo != 0) & (hi != 0)
    # the faces west, east, south, north of a cell: the sides whose higher
    # (lower) cell it is
    faces = [(vertical & (hi != 0), hi), (vertical & (lo != 0), lo), (~vertical & (hi != 0), hi),
             (~vertical & (lo != 0), lo)]
    faces[0][0][0] = faces[1][0][0] = faces[2][0][0] = faces[3][0][0] = False
    faces = [(m.nonzero()[:, 0], c[m]) for m, c in faces]

    def face(values, d):
        ids, cell = faces[d]
        return torch.zeros(e, dtype=torch.float64, device=dev).index_add_(0, cell, values[ids])

    depth = put(w.initial_depth)
    depth = torch.where(level_cell, (start - bed).clamp(min=0), depth)
    depth[0] = 0
    q = torch.zeros(a.s_num, dtype=torch.float64, device=dev)
    rain_time, infiltration = torch.zeros_like(depth), torch.zeros_like(depth)
    max_depth, max_speed = depth.clone(), torch.zeros_like(depth)
    infiltration = f0.clone() if w.initial_depth is None else infiltration
    theta = float(np.float32(w.sita))
    face_length = [face(length, d) for d in range(4)] if theta != 1 else None
    opened = put(a.open_face) if theta != 1 else None
    hang = put(a.hcells) if a.hang_cells else None

    def gradients():
        """Tangential surface gradient of the cells beside hanging edges."""
        wet, eta = depth > min_h, bed + depth
        out = torch.zeros(len(hang), 2, dtype=torch.float64, device=dev)
        axes = put(a.axes)
        for axis in (0, 1):
            found = []
            for d in (2 * axis, 2 * axis + 1):
                ids, cell = faces[d]
                other = lo[ids] + hi[ids] - cell
                use = ((other != 0) & wet[other]).double() * length[ids]
                bad = face_of(ids, cell, 1.0 - (use > 0).double())
                total = face_of(ids, cell, use)
                span = (y[other] - y[cell]) if axis else (x[other] - x[cell])
                value = face_of(ids, cell, use * (eta[other] - eta[cell]))[hang] / total[hang].clamp(min=1e-30)
                reach = face_of(ids, cell, use * span)[hang] / total[hang].clamp(min=1e-30)
                found.append((value, reach, (total[hang] > 0) & (bad[hang] == 0)))
            (vm, xm, om), (vp, xp, op) = found
            one = torch.ones_like(vm)
            both = (vp - vm) / torch.where(om & op, xp - xm, one)
            left, right = vm / torch.where(om, xm, one), vp / torch.where(op, xp, one)
            got = torch.where(om & op, both, torch.where(om, left, torch.where(op, right, 0 * one)))
            out[:, axis] = torch.where((axes[:, axis] == 1) & wet[hang], got, 0 * got)
        return out

    def face_of(ids, cell, values):
        return torch.zeros(e, dtype=torch.float64, device=dev).index_add_(0, cell, values)

    def neighbours():
        """Sum of the discharges of the faces beyond a side's two cells, with
        the open-face rule at open boundaries."""
        mean = torch.stack([face(q * length, d) / face_length[d].clamp(min=1e-30) for d in range(4)], 1)
        below, above = torch.where(vertical, 0, 2), torch.where(vertical, 1, 3)
        left, right = mean[lo, below], mean[hi, above]
        lext, rext = opened[lo, below], opened[hi, above]
        product = lext * rext
        mixed = (((1 - rext) * left + (1 - lext) * right + 2 * q * (lext + rext - 2 * product))
                 / torch.where(product == 1, torch.ones_like(product), 1 - product))
        whole = (lext == 1) | (rext == 1)
        return torch.where((lext > 0) | (rext > 0), torch.where(whole, 2 * q, mixed), left + right)

    def face_depth():
        return torch.maximum(bed[lo] + depth[lo], bed[hi] + depth[hi]) - torch.maximum(bed[lo], bed[hi]).clamp(min=dh)

    def courant():
        h = face_depth().clamp(min=0.01)
        return float((w.afa * length / ((G * h).sqrt() + q.abs() / h))[inner].min())

    elapsed, u, v = 0.0, None, None
    step = courant()
    for _ in range(BATCH):
        dt = min(step, 1.0)
        wh = face_depth()
        difference = bed[hi] + depth[hi] - bed[lo] - depth[lo]
        if hang is not None:
            grad, index = gradients(), put(a.edge_index)
            ids = ((index >= 0) & (depth[lo] > min_h) & (depth[hi] > min_h)).nonzero()[:, 0]
            at, axis = index[ids], vertical[ids].long()
            offsets, slots = put(a.offsets).reshape(-1, 2)[at], put(a.slots).reshape(-1, 2)[at]
            difference[ids] += (torch.where(offsets[:, 1] != 0, grad[slots[:, 1], axis] * offsets[:, 1], 0.0)
                                - torch.where(offsets[:, 0] != 0, grad[slots[:, 0], axis] * offsets[:, 0], 0.0))
        push = -G * difference / dx * wh.clamp(min=0) * dt
        friction = 1 + G * dt * n * n * (q / wh.clamp(min=1e-5) ** (7.0 / 3.0)).abs()
        beside = neighbours() if theta != 1 else 0.0
        new = (theta * q + (1 - theta) / 2 * beside + push) / friction
        q = torch.where((wh < min_h) | closed, torch.zeros_like(new), new)
        q[0] = 0
        volume = q * length
        out = sum(face((-volume if d in (0, 2) else volume).clamp(min=0) * dt, d) for d in range(4))
        available = depth * area + rate * dt * area
        scale = torch.where((out > available) & ~level_cell, available / out.clamp(min=1e-30), torch.ones_like(out))
        scale[0] = 0
        q = q * scale[torch.where(q >= 0, lo, hi)]
        raining = rate > 0
        rain_time = torch.where(raining, rain_time + dt, rain_time)
        infiltration = torch.where(raining, fc + (f0 - fc) * torch.exp(-k * rain_time / 3600.0), infiltration)
        west, east, south, north = (face(q * length, d) for d in range(4))
        raw = depth + (west - east + south - north) * dt / area.clamp(min=1e-30) + rate * dt
        raw = raw - torch.minimum(infiltration * dt, raw.clamp(min=0))
        elapsed += dt
        depth = torch.where(level_cell, (start + slope * elapsed - bed).clamp(min=0), raw.clamp(min=0))
        depth[0] = 0
        wet, h = depth >= min_h, depth.clamp(min=0.01)
        u = torch.where(wet, (west + east) / height.clamp(min=1e-30) / h / 2, 0 * h)
        v = torch.where(wet, (south + north) / width.clamp(min=1e-30) / h / 2, 0 * h)
        max_speed = torch.maximum(max_speed, (u * u + v * v).sqrt())
        max_depth = torch.maximum(max_depth, depth)
        step = courant()
    return dict(depth=depth, q=q, rain_time=rain_time, infiltration=infiltration, max_depth=max_depth,
                max_speed=max_speed, u=u, v=v, peak_ticks=[None, None], steps=None, elapsed=elapsed)
