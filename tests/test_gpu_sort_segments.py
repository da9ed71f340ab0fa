"""The sort's long segments (cells of more than 64 particles) against a stable argsort: from a random
order, from the order a push left (nearly all of a cell's slots from one work unit, a few from
others), with products appended past the sorted slots, and with cells spread over several work
units.  Integer work: the order must be identical."""
import numpy as np
import pytest

from jd_lepic_b200 import configs

pytestmark = pytest.mark.gpu


def _expected(p, case, tile):
    cx = np.floor(p[:, 0] / case.dx + 1e-9).astype(int)
    cy = np.floor(p[:, 1] / case.dy + 1e-9).astype(int)
    tx, ty = cx // tile, cy // tile
    ntx = -(-case.nx // tile)
    key = ((ty * ntx + tx) * tile + cy % tile) * tile + cx % tile
    return p[np.argsort(key, kind="stable")]


@pytest.mark.parametrize("n", [3000, 60000, 400000])
@pytest.mark.parametrize("cells", [(8, 8), (24, 16), (5, 3)])
def test_long_segments_are_stable(gpu_lib, cells, n):
    from jd_lepic_b200.simulation import GpuSimulation
    nx, ny = cells
    tile = 4
    case = configs.case0(ppc=1, nx=nx, ny=ny)
    case.ng = 1
    s = GpuSimulation(case, tile=(tile, tile), load=False, capacity=n + 8)
    try:
        rng = np.random.default_rng(n + nx)
        p = np.zeros((n, 6))
        p[:, 0] = (0.5 + rng.random(n) * (nx - 1)) * case.dx
        p[:, 1] = (0.5 + rng.random(n) * (ny - 1)) * case.dy
        p[: n // 2, :2] = 0.3 * p[: n // 2, :2]                 # a dense corner
        p[:, 3:5] = rng.normal(0, 0.05 * case.dx / case.dt, (n, 2))
        s.put_particles(0, p)
        s.set_phi(np.zeros((ny + 3, nx + 3)))
        s.efield()
        for it in range(1, 6):
            before = s.get_particles(0)
            s.sort(0)
            got = s.get_particles(0)
            assert np.array_equal(got, _expected(before, case, tile))
            for k in range(1 + it % 3):
                s.push(10 * it + k)
    finally:
        s.close()


@pytest.mark.parametrize("spread", [0.0, 0.3])
def test_segments_with_an_appended_tail(gpu_lib, spread):
    """Particles put after a sort (the occupied slots replaced) and duplicated behind the sorted ones:
    the next sort meets the old units and a tail in one segment."""
    from jd_lepic_b200.simulation import GpuSimulation
    n = 20000
    case = configs.case0(ppc=1, nx=6, ny=6)
    case.ng = 1
    s = GpuSimulation(case, tile=(2, 2), load=False, capacity=4 * n)
    try:
        rng = np.random.default_rng(3)
        p = np.zeros((n, 6))
        p[:, :2] = (0.5 + rng.random((n, 2)) * 5) * case.dx
        p[:, 3:5] = rng.normal(0, spread * case.dx / case.dt, (n, 2))
        for sp in range(2):
            s.put_particles(sp, p)
            s.sort(sp)
        s.set_phi(np.zeros((9, 9)))
        s.efield()
        s.push(1)
        s.check(s.lib.lepic_gpu_duplicate_particles(s.ctx, 2), "duplicate")
        before = s.get_particles(0)
        s.sort(0)
        assert np.array_equal(s.get_particles(0), _expected(before, case, 2))
    finally:
        s.close()
