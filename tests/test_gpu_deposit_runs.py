"""The deposit through per-run moments against the integer CIC restated in numpy, bit for bit: the
context's accumulators and lepic_gpu_deposit_noalloc's grid, on grids whose products of the
fixed-point offsets are rounded by 4 bits, by 2, not at all and shifted up (S = 24, 23, 22, 21),
with particles in cell order, in random order, alone in their cells, on cell edges, and in
numbers around a thread's share."""
import ctypes as C

import numpy as np
import pytest

from jd_lepic_b200 import _capi as capi, configs
from oracle import oracle as O
from test_gpu_decomposition import _acc_view, _fixed_point

pytestmark = pytest.mark.gpu

SIZES = [(40, 56), (256, 200), (511, 33), (1024, 24), (2048, 16)]   # S = 24, 24, 23, 22, 21


@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("size", SIZES)
def test_context_accumulators_are_exact(gpu_lib, size, sort):
    from jd_lepic_b200.simulation import GpuSimulation
    nx, ny = size
    case = configs.case0(ppc=1, nx=nx, ny=ny)
    case.ng = 1
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=80000)
    try:
        rng = np.random.default_rng(nx)
        for n in (1, 3, 70001):
            p = np.zeros((n, 6))
            p[:, 0] = rng.random(n) * nx * case.dx * 0.9999
            p[:, 1] = rng.random(n) * ny * case.dy * 0.9999
            p[::7, 0] = np.floor(p[::7, 0] / case.dx) * case.dx      # on a cell edge
            p[:n // 3, :2] = p[0, :2] * np.array([1.0, 1.0])         # many in one place
            s.put_particles(0, p)
            if sort:
                s.sort(0)
            s.deposit()
            X, Y, S = _fixed_point(s, 0)
            ref = O.int_deposit(X, Y, nx, ny, S).view(np.int64)
            assert np.array_equal(_acc_view(s, 0).cpu().numpy(), ref)
    finally:
        s.close()


@pytest.mark.parametrize("order", ["sorted", "random"])
@pytest.mark.parametrize("size", SIZES)
def test_noalloc_is_exact(gpu_lib, size, order):
    import torch
    nx, ny = size
    S = min(24, 32 - int(np.ceil(np.log2(max(nx, ny)))))
    nn = (nx + 3) * (ny + 3)
    rng = np.random.default_rng(ny)
    kq = torch.from_numpy(rng.integers(1, 3, nn).astype(np.float64)).cuda()
    # the largest (where weights are rounded): several passes of the whole grid of warps, and in cell
    # order every warp's 128 slots in one cell or two: the packed counts and remainder sums at their largest
    large = ((20000003, 0), (20000003, 1)) if size in ((40, 56), (511, 33)) else ()
    small = 1 << 19                           # one slot per lane up to here, four beyond
    for n, lead in ((1, 0), (5, 1), (1023, 3), (200003, 0), (200003, 2), (small, 1), (small + 1, 3), (3000017, 0)) + large:
        X = rng.integers(0, nx << S, n, dtype=np.int64)
        Y = rng.integers(0, ny << S, n, dtype=np.int64)
        if order == "sorted":
            o = np.argsort((Y >> S) * nx + (X >> S), kind="stable")
            X, Y = X[o], Y[o]
        VX = rng.normal(size=n).astype(np.float32)
        VX[rng.random(n) < 0.05] = np.nan
        live = ~np.isnan(VX)
        X2, Y2 = X.copy(), Y.copy()
        out_of_box = rng.random(n) < 0.01
        if nx << S < 1 << 32:                     # positions past the box are skipped
            X2[out_of_box] = (nx << S) + 5
            live &= ~out_of_box
        dev = []
        for a in (X2.astype(np.uint32).view(np.int32), Y2.astype(np.uint32).view(np.int32), VX):
            t = torch.zeros(n + 8, dtype=torch.from_numpy(a).dtype, device="cuda")
            t[lead:lead + n] = torch.from_numpy(a)    # lead: arrays that are not 16-byte aligned
            dev.append(t)
        out = torch.full((nn,), float("nan"), dtype=torch.float64, device="cuda")
        k1 = 0.37
        ptr = [C.c_void_p(t.data_ptr() + 4 * lead) for t in dev]
        rc = gpu_lib.lepic_gpu_deposit_noalloc(ptr[0], ptr[1], ptr[2], n, nx, ny, S, k1, C.c_void_p(kq.data_ptr()),
                                               C.c_void_p(out.data_ptr()),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == capi.OK
        acc = O.int_deposit(X[live], Y[live], nx, ny, S)
        ref = kq.cpu().numpy() * (k1 * (acc.astype(np.float64) * 2.0 ** -44))
        assert np.array_equal(out.cpu().numpy(), ref)
