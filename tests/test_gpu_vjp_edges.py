"""The vector-Jacobian products at the sizes where their tiles end: lists of 32 and 64 entries and
groups of 32 bodies in the tree's, turns of 64 and tiles of 512 bodies in the symmetric pairwise one.
Against the one-sided pairwise kernel, with the tolerances of the larger comparisons (test_gpu_adjoint.py):
FP32 rounding of sums over the same pairs in another order."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from lettuce_simulate_physics_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    with L.CudaBackend(0) as b:
        yield b


def gradients(be, b, method, mode, monkeypatch):
    monkeypatch.setenv("LETTUCE_GB300_VJP", mode)
    be.upload(b)
    be.adjoint_forward(L.ForceParams(G=1.0, eps=0.05, theta=0.0, method=method), 1e-2, 3, 2)
    return be.adjoint_backward(b.pos64() + 0.01)


def same(got, want, tol):
    assert abs(got[0] - want[0]) <= 1e-6 * abs(want[0])
    for g, w in zip(got[1:], want[1:]):
        assert np.isfinite(g).all()
        assert np.linalg.norm(g - w) <= tol * np.linalg.norm(w)


@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129, 300])
def test_tree(be, n, monkeypatch):
    b = S.cube(n, n)
    want = gradients(be, b, L.ForceMethod.direct, "pairs", monkeypatch)
    same(gradients(be, b, L.ForceMethod.tree, "pairs", monkeypatch), want, 1e-5)


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 511, 512, 513, 1024, 1025])
def test_symmetric(be, n, monkeypatch):
    b = S.cube(n, n)
    want = gradients(be, b, L.ForceMethod.direct, "pairs", monkeypatch)
    same(gradients(be, b, L.ForceMethod.direct, "symmetric", monkeypatch), want, 2e-6)
