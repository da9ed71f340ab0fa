"""The FP64 multigrid's execution paths against the CPU restatement: levels swept in shared-memory
tiles (every level with mg_small_nodes = 0), levels held by one CTA, both together and the whole
problem in one CTA, on grids whose sides are no multiples of a tile, narrow and wide ones, with an
embedded plate, a Neumann column and periodic edges (an odd number of rows on the coarsest level
included).  The paths run the reference's operations in the reference's order: the same cycle
and sweep counts, and phi to 1e-13 of its maximum."""
import ctypes as C

import numpy as np
import pytest

from jd_lepic_b200 import _capi as capi, configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(nx, ny, ng, kind):
    case = configs.case0(ppc=1, nx=nx, ny=ny)
    case.ng = ng
    b = configs.box_mask(nx, ny, label_left=1, label_right=2)
    if "pbc" in kind:
        b[0:2, 2:nx + 1] = 0
        b[ny + 1:, 2:nx + 1] = 0
        case.flag_pbc = 1
    if "nmn" in kind:
        b[slice(0, ny + 3) if "pbc" in kind else slice(2, ny + 1), 0:2] = -2
        case.flag_nmn = 1
    if "plate" in kind:
        x = nx // 2 + 1
        b[2 + ny // 4:2 + ny // 2, x:x + max(2, nx // 8)] = 3
    case.bcnd = b
    case.phi0 = configs.potentials(b, {1: 0.0, 2: 10.0, 3: -20.0})
    return case


# (nx, ny, levels, boundaries): sizes around a tile's edge, odd factors, flat and tall boxes
GRIDS = [(96, 48, 5, "box"), (40, 136, 4, "plate"), (24, 200, 4, "pbc"), (72, 88, 4, "pbc_nmn"), (132, 20, 3, "nmn"),
         (36, 12, 3, "pbc"), (128, 128, 7, "plate"), (33, 47, 1, "box"), (260, 196, 3, "pbc_plate"),
         # an odd number of columns over an even number of rows on a level that one CTA holds
         (96, 64, 6, "box"), (33, 20, 1, "box"), (48, 64, 5, "pbc")]


@pytest.mark.parametrize("small", [0, 300, 2000, 5000])
@pytest.mark.parametrize("grid", GRIDS)
def test_paths_match_oracle(gpu_lib, grid, small):
    from jd_lepic_b200.simulation import GpuSimulation
    nx, ny, ng, kind = grid
    case = _case(nx, ny, ng, kind)
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=64)
    try:
        s.set_options(mg_small_nodes=small)
        rng = np.random.default_rng(nx + ny)
        X, Y = np.meshgrid(np.arange(nx + 1) / nx, np.arange(ny + 1) / ny)
        rhs = 1.6e-3 * np.sin(3 * np.pi * X) * np.cos(2 * np.pi * Y) + 2e-4 * rng.normal(size=X.shape)
        a = np.ascontiguousarray(rhs)
        s.check(s.lib.lepic_gpu_set_grid(s.ctx, capi.GRID_RHS, a.ctypes.data_as(C.POINTER(C.c_double))), "set_grid")
        st = s.solve(eps=1e-9, mode=capi.POISSON_FP64_MG, phi=case.phi0.copy())
        ref = case.phi0.copy()
        rc, ost = O.solve(O.make_cfg(case, s.sp), ref, rhs, case.bcnd, ng, 1e-9)
        assert rc == 0
        assert (st["cycles"], st["sweeps_fine"]) == (ost.k, ost.sweeps_fine)
        assert np.abs(st["phi"] - ref).max() <= 1e-13 * np.abs(ref).max()
        # the relative L2 criterion from the same start: its residual as the oracle measures it
        st2 = s.solve(eps=1e-7, mode=capi.POISSON_FP64_MG_L2, phi=case.phi0.copy())
        l2 = O.l2_residual(O.make_cfg(case, s.sp), st2["phi"], rhs, case.bcnd)
        assert l2 <= 1e-7 and abs(l2 - st2["res_l2_rel"]) <= 1e-6 * l2 + 1e-15
    finally:
        s.close()


@pytest.mark.parametrize("small", [0, 300, 2000])
@pytest.mark.parametrize("size", [(32, 24, 3), (64, 48, 4), (96, 72, 4)])
def test_free_right_column_between_periodic_edges(gpu_lib, size, small):
    """Free nodes in the right column of a periodic deck: the restriction of the bottom row asks for
    a residual one node past the grid, which counts as zero on every path."""
    from jd_lepic_b200.simulation import GpuSimulation
    nx, ny, ng = size
    case = _case(nx, ny, ng, "pbc")
    case.bcnd[:, nx + 1:] = 0
    case.phi0 = configs.potentials(case.bcnd, {1: 5.0})
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=64)
    try:
        s.set_options(mg_small_nodes=small)
        rng = np.random.default_rng(nx)
        X, Y = np.meshgrid(np.arange(nx + 1) / nx, np.arange(ny + 1) / ny)
        rhs = 1.6e-3 * np.sin(3 * np.pi * X) * np.cos(2 * np.pi * Y) + 2e-4 * rng.normal(size=X.shape)
        a = np.ascontiguousarray(rhs)
        s.check(s.lib.lepic_gpu_set_grid(s.ctx, capi.GRID_RHS, a.ctypes.data_as(C.POINTER(C.c_double))), "set_grid")
        st = s.solve(eps=1e-9, mode=capi.POISSON_FP64_MG, phi=case.phi0.copy())
        ref = case.phi0.copy()
        rc, ost = O.solve(O.make_cfg(case, s.sp), ref, rhs, case.bcnd, ng, 1e-9)
        assert rc == 0 and ost.k < 20
        assert (st["cycles"], st["sweeps_fine"]) == (ost.k, ost.sweeps_fine)
        assert np.abs(st["phi"] - ref).max() <= 1e-13 * np.abs(ref).max()
    finally:
        s.close()


@pytest.mark.parametrize("small", [0, 300, 2000])
@pytest.mark.parametrize("size", [(32, 24, 3), (64, 48, 4), (96, 72, 4)])
def test_counted_nodes_on_the_copied_edge_row(gpu_lib, size, small):
    """Label -1 on the upper edge row of a periodic deck: its nodes' residuals count, and the copy of
    row 1 overwrites them after each half-sweep.  They never vanish, so the cycles run out; residual
    and potential are the restatement's."""
    from jd_lepic_b200.simulation import GpuSimulation
    nx, ny, ng = size
    case = _case(nx, ny, ng, "pbc")
    case.bcnd[ny + 1, 2:nx + 1] = -1
    case.phi0 = configs.potentials(case.bcnd, {1: 5.0, 2: 10.0})
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=64, config={"ncycl": 6})
    try:
        s.set_options(mg_small_nodes=small)
        rng = np.random.default_rng(nx)
        X, Y = np.meshgrid(np.arange(nx + 1) / nx, np.arange(ny + 1) / ny)
        rhs = 1.6e-3 * np.sin(3 * np.pi * X) * np.cos(2 * np.pi * Y) + 2e-4 * rng.normal(size=X.shape)
        a = np.ascontiguousarray(rhs)
        s.check(s.lib.lepic_gpu_set_grid(s.ctx, capi.GRID_RHS, a.ctypes.data_as(C.POINTER(C.c_double))), "set_grid")
        s.set_phi(case.phi0)
        st = capi.LepicSolveStats()
        rc = s.lib.lepic_gpu_iterative_solver(s.ctx, None, 0.02, capi.POISSON_FP64_MG, C.byref(st))
        ref = case.phi0.copy()
        orc, ost = O.solve(O.make_cfg(case, s.sp), ref, rhs, case.bcnd, ng, 0.02, ncycl=6)
        assert rc == capi.ENOTCONV and orc == 0 and ost.k == 6
        assert (st.cycles, st.sweeps_fine) == (ost.k, ost.sweeps_fine)
        assert abs(st.res_l1 - ost.res) <= 1e-12 * ost.res
        assert np.abs(s.grid(capi.GRID_PHI) - ref).max() <= 1e-13 * np.abs(ref).max()
    finally:
        s.close()


# cell sizes (m) with unrelated mantissas of the diagonal, one whose diagonal lies above 1e30 on all
# levels but the coarsest, one below 1e-30 on all of them: there the general division takes every dividend
CELLS = [(1e-4, 1e-4, (1e-300, 1e-150, 1.0, 1e150, 1e280)), (1.371e-4, 0.733e-4, (1e-300, 1.0, 1e280)),
         (3.1e-5, 2.9e-5, (1e-150, 1.0, 1e272)), (1e-21, 1.3e-21, (1e-150, 1.0, 1e150)), (1e10, 1.7e10, (1e-150, 1.0, 1e150))]


@pytest.mark.parametrize("cell", CELLS)
def test_quotient_of_extreme_values(gpu_lib, cell):
    """The update divides by the fixed diagonal with a corrected reciprocal where dividend and
    diagonal are in range (2^-899 to 2^901, 1e-30 to 1e30) and with the general division elsewhere:
    sources from 1e-300 to 1e280 beside nodes that are zero, bit for bit."""
    from jd_lepic_b200.simulation import GpuSimulation
    nx = ny = 32
    case = _case(nx, ny, 4, "box")
    case.dx, case.dy = cell[0], cell[1]
    case.phi0 = np.zeros_like(case.phi0)
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=64, config={"ncycl": 1})
    try:
        for scale in cell[2]:
            rhs = np.zeros((ny + 1, nx + 1))
            rhs[5, 7], rhs[20, 11] = scale, -3.0 * scale
            a = np.ascontiguousarray(rhs)
            s.check(s.lib.lepic_gpu_set_grid(s.ctx, capi.GRID_RHS, a.ctypes.data_as(C.POINTER(C.c_double))), "set_grid")
            s.set_phi(case.phi0)
            rc = s.lib.lepic_gpu_iterative_solver(s.ctx, None, 1e-320, capi.POISSON_FP64_MG, None)
            assert rc == 0
            assert s.lib.lepic_gpu_sync(s.ctx) in (0, capi.ENOTCONV)
            got = s.grid(capi.GRID_PHI)
            ref = case.phi0.copy()
            O.solve(O.make_cfg(case, s.sp), ref, rhs, case.bcnd, 4, 1e-320, ncycl=1)
            assert np.isfinite(ref).all() and np.abs(ref).max() > 0.0
            assert np.array_equal(got, ref)
    finally:
        s.close()
