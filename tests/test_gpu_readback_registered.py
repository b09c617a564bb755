"""Readbacks into columns of one buffer of which only some are page-locked, or each by itself: a copy must
not reach from one into the next."""
import mmap

import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "m", "id")


@pytest.mark.parametrize("locked", [(0,), (1,), (2,), (0, 1), (0, 2), (1, 2, 3), (0, 1, 2, 3, 4, 5, 6, 7), (4, 7)])
@pytest.mark.parametrize("pages", [1, 40])
def test_columns_locked_one_by_one(locked, pages):
    torch = pytest.importorskip("torch")
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    size = pages * mmap.PAGESIZE  # of a column: whole pages
    n = size // 4
    rng = np.random.Generator(np.random.PCG64(n))
    b = L.Bodies(*(rng.normal(size=n).astype(np.float32) for _ in range(7)), rng.permutation(n).astype(np.uint32))
    with L.CudaBackend(0) as be:
        be.upload(b)
        be.compute_forces(L.ForceParams(G=1.0, eps=0.1, theta=0.9, method=L.ForceMethod.tree), True)
        b, a = be.download(), be.accel()
        memory = mmap.mmap(-1, 8 * size)
        cols = [np.frombuffer(memory, np.float32 if k < 7 else np.uint32, n, k * size) for k in range(8)]
        rt = torch.cuda.cudart()
        torch.cuda.init()
        for k in locked:
            assert int(rt.cudaHostRegister(cols[k].ctypes.data, size, 0)) == 0
        try:
            out = be.download(L.Bodies(*cols))
            for f in FIELDS:
                assert np.array_equal(getattr(out, f), getattr(b, f)), f
            ptr = [c.ctypes.data_as(L.backend._f) for c in cols[:4]]
            L.backend._check(be._lib.lg_read_accel(be._h, *ptr))
            assert np.array_equal(np.stack(cols[:4]), a)
        finally:
            for k in locked:
                rt.cudaHostUnregister(cols[k].ctypes.data)
