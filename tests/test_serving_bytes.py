"""Device bytes of a served solve, for the step forms that the server's engines
choose: the estimate covers what creating the solve takes on the device, without
much to spare, and the bound taken before its arrays exist covers the estimate."""
import pytest

from test_gpu_resident import grid, quadtree

MESHES = {
    'lattice': lambda: grid(1400, 1300),
    'lattice_horton_rows': lambda: grid(1250, 1111, horton=True, rows=True),
    'lattice_flat': lambda: grid(300, 4000),
    'lattice_small': lambda: grid(640, 500, horton=True),
    'below_the_lattice': lambda: grid(400, 500),
    'theta': lambda: grid(600, 600, theta=0.8),
    'quadtree': lambda: quadtree(9000),
}


@pytest.mark.parametrize('name', sorted(MESHES))
def test_bound_covers_estimate(name):
    from nhflood.serving import device_bytes_bound, device_bytes_estimate
    w = MESHES[name]()
    assert device_bytes_bound(w) >= device_bytes_estimate(w.step_arrays())


def test_lattice_counts_from_its_size_on():
    """A uniform grid that runs on the lattice holds at least the march's maps and
    state copies; one with theta < 1 or fewer cells runs on tiles."""
    from nhflood.serving import device_bytes_estimate, tiled_bytes
    for make, lattice in (('lattice_small', True), ('below_the_lattice', False), ('theta', False)):
        arrays = MESHES[make]().step_arrays()
        e, s = arrays.e_num, arrays.s_num
        rest = arrays.nbytes() + 4 * (10 * e + s) + 4 * (s + 5 * e) + 16 * ((e + 255) // 256) * arrays.terms
        form = device_bytes_estimate(arrays) - rest - (1 << 20)
        assert (form > 91 * e) == lattice and form >= tiled_bytes(e, s), make


@pytest.mark.gpu
@pytest.mark.parametrize('name', sorted(MESHES))
def test_estimate_covers_the_device(cuda_available, name):
    """Torch and the driver give memory in pieces of 2 MB, some 40 of them here."""
    import torch
    from nhflood.ensemble import plain_factory
    from nhflood.plain import PlainRun
    from nhflood.serving import device_bytes_estimate
    w = MESHES[name]()
    arrays = w.step_arrays()
    PlainRun(grid(40, 33), plain_factory()).close()      # the context and the kernels are there
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    run = PlainRun(w, plain_factory(), arrays=arrays)
    assert run.engine.path.startswith('lattice') == name.startswith('lattice'), run.engine.path
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    used = before - torch.cuda.mem_get_info()[0]
    estimate = device_bytes_estimate(arrays)
    assert used <= estimate + 80 * (1 << 20), (name, used / arrays.e_num, estimate / arrays.e_num)
    assert estimate <= 1.25 * used + 80 * (1 << 20), (name, used / arrays.e_num, estimate / arrays.e_num)
    run.close()
