"""Particles put from and read back to the host across the staging chunks (131072 particles): positions
on the fixed-point grid as llround places them, FP32 velocities, the order kept, holes left out,
and a refused call leaving the species as it was."""
import ctypes as C

import numpy as np
import pytest

from jd_lepic_b200 import _capi as capi, configs

pytestmark = pytest.mark.gpu

CHUNK = 131072     # the largest chunk; several host threads and pinned buffers from 8 of them on


def _particles(case, n, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros((n, 6))
    p[:, 0] = rng.random(n) * case.nx * case.dx * (1 - 1e-6)
    p[:, 1] = rng.random(n) * case.ny * case.dy * (1 - 1e-6)
    p[:, 3:] = rng.normal(0, 1e6, (n, 3))
    return p


def _stored(p, case):
    S = min(24, 32 - int(np.ceil(np.log2(max(case.nx, case.ny)))))
    q = p.copy()
    for k, h in ((0, case.dx), (1, case.dy)):
        q[:, k] = np.floor(p[:, k] * (2.0 ** S / h) + 0.5) * (h * 2.0 ** -S)
    q[:, 2] = 0.0
    q[:, 3:] = p[:, 3:].astype(np.float32)
    return q


@pytest.mark.parametrize("n", [0, 1, 1023, CHUNK - 1, CHUNK, CHUNK + 1, 2 * CHUNK + 5, 5 * CHUNK - 700,
                               8 * CHUNK - 1, 8 * CHUNK, 13 * CHUNK + 700])
def test_round_trip(gpu_lib, n):
    from jd_lepic_b200.simulation import GpuSimulation
    case = configs.case0(ppc=1, nx=64, ny=48)
    case.ng = 1
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=max(1, n))
    try:
        for seed in (n, n + 1):                       # twice: the buffers take turns
            p = _particles(case, n, seed)
            s.put_particles(0, p)
            assert np.array_equal(s.get_particles(0), _stored(p, case))
            st = s.push_stats()
            assert st["np_tot"][0] == n and st["n_slots"][0] == n
        if n:
            # a velocity that is no number marks a hole, left out of the read
            q = p.copy()
            q[::3, 3] = np.nan
            s.put_particles(0, q)
            assert np.array_equal(s.get_particles(0), _stored(q[~np.isnan(q[:, 3])], case))
            # too small an output: the first ones, and the code
            kept = s.get_particles(0)
            m = C.c_int64()
            out = np.full((len(kept) + 1, 6), -1.0)
            cap = max(0, len(kept) - 2)
            rc = s.lib.lepic_gpu_get_particles(s.ctx, 0, out.ctypes.data_as(C.POINTER(C.c_double)), cap, C.byref(m))
            assert rc == (capi.ECAPACITY if len(kept) else capi.OK) and m.value == len(kept)
            assert np.array_equal(out[:cap], kept[:cap]) and np.all(out[cap:] == -1.0)
    finally:
        s.close()


@pytest.mark.parametrize("size", [2, 8])
@pytest.mark.parametrize("at", [0, CHUNK - 1, 2 * CHUNK + 3])
@pytest.mark.parametrize("what", [(0, -1e-4), (1, 1.0), (0, np.nan), (1, np.inf)])
def test_refused_put_changes_nothing(gpu_lib, at, what, size):
    from jd_lepic_b200.simulation import GpuSimulation
    case = configs.case0(ppc=1, nx=32, ny=32)
    n = size * CHUNK + 10
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=n)
    try:
        p = _particles(case, 5000, 1)
        s.put_particles(0, p)
        s.sort(0)
        before = s.get_particles(0)
        bad = _particles(case, n, 2)
        bad[at, what[0]] = what[1]
        with pytest.raises(capi.LepicError) as e:
            s.put_particles(0, bad)
        assert e.value.code == capi.EINVAL
        assert np.array_equal(s.get_particles(0), before)
        s.sort(0)
        assert np.array_equal(s.get_particles(0), before)
    finally:
        s.close()


@pytest.mark.parametrize("n", [1, 5000, CHUNK + 1, 8 * CHUNK])
def test_arrays_in_use_show_a_put(gpu_lib, n):
    """Pointers taken before a put show the particles put, those of a refused one the old ones."""
    import torch

    class Dev:
        def __init__(self, ptr, kind):
            self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False), "version": 2}

    from jd_lepic_b200.simulation import GpuSimulation
    case = configs.case0(ppc=1, nx=32, ny=32)
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=n)
    try:
        s.put_particles(0, _particles(case, n, 3))
        for sort in (False, True):
            if sort:
                s.sort(0)                             # goes over to the other arrays
            ptr = [C.c_void_p() for _ in range(5)]
            s.check(s.lib.lepic_gpu_particle_arrays(s.ctx, 0, *[C.byref(v) for v in ptr], None, None), "particle_arrays")
            p = _particles(case, n, 4)
            p[::5, 3] = np.nan
            s.put_particles(0, p)
            bad = _particles(case, n, 5)
            bad[n - 1, 0] = -1.0
            with pytest.raises(capi.LepicError):
                s.put_particles(0, bad)
            got = [torch.as_tensor(Dev(v.value, "<i4" if q < 2 else "<f4"), device="cuda").cpu().numpy()
                   for q, v in enumerate(ptr)]
            for k, h in ((0, case.dx), (1, case.dy)):
                assert np.array_equal(got[k].view(np.uint32), np.floor(p[:, k] * (2.0 ** 24 / h) + 0.5).astype(np.uint32))
            for k in range(3):
                assert np.array_equal(got[2 + k], p[:, 3 + k].astype(np.float32), equal_nan=True)
    finally:
        s.close()


@pytest.mark.parametrize("capacity", [1024, 20000, CHUNK, 700000])
def test_full_species_crosses_in_large_chunks(gpu_lib, capacity):
    """A species as large as the sort's scratch allows, put, sorted and read back: the scratch holds a
    chunk of up to 131072 particles beside the read's block offsets."""
    from jd_lepic_b200.simulation import GpuSimulation
    case = configs.case0(ppc=1, nx=48, ny=40)
    case.ng = 1
    s = GpuSimulation(case, tile=(8, 8), load=False, capacity=capacity)
    try:
        p = _particles(case, capacity, 9)
        s.put_particles(0, p)
        s.put_particles(1, p[::-1])
        s.sort(0)
        assert np.array_equal(s.get_particles(1), _stored(p[::-1], case))
        a, b = s.get_particles(0), _stored(p, case)
        assert np.array_equal(a[np.lexsort(a.T)], b[np.lexsort(b.T)])
    finally:
        s.close()
