"""Leaves of coincident bodies in the walks' lists: more than 16 bodies each, they enter a packet (768
bodies, 256 ranges) one range at a time, split where it is full, among the short ranges of other
leaves. Hundreds of them of every length fill packets at every place. At theta 0 all pairs are taken as
bodies; against the FP64 direct sum (tolerances of test_gpu_walk.py) and, for the adjoint, the
pairwise product (test_gpu_vjp_edges.py)."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from gpu_util import by_id, params, rel_rms, zero_v
from lettuce_simulate_physics_gb300 import scenarios as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EPS = 0.05


@pytest.fixture(scope="module")
def be():
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    with L.CudaBackend(0) as b:
        yield b


def clumps(lengths, single, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    p = np.concatenate([np.repeat(rng.uniform(-1, 1, (len(lengths), 3)), lengths, axis=0), rng.uniform(-1, 1, (single, 3))])
    p = p[rng.permutation(len(p))]
    z = np.zeros(len(p))
    return L.Bodies(*p.T, z, z, z, rng.uniform(0.5, 1.5, len(p)) / len(p), np.arange(len(p)))


CASES = [((17,) * 200, 900), (tuple(range(17, 90)), 0), ((255, 256, 257, 511, 767, 768, 769), 333), ((18,) * 45, 40),
         (tuple(17 + (7 * k) % 40 for k in range(150)), 2000)]


@pytest.mark.parametrize("lengths,single", CASES)
def test_forces(be, lengths, single):
    b = clumps(list(lengths), single, len(lengths))
    n = len(b)
    exact = O.direct_fp64(b, 1.0, EPS)
    be.upload(zero_v(b))
    for _ in range(2):
        be.compute_forces(params(1, EPS, 0.0), True)
        a = by_id(be.download().id, be.accel())
        assert be.times().interactions == n * (n - 1)
        assert rel_rms(a[:3], exact[:3]) <= 2e-6
        np.testing.assert_allclose(a[3], exact[3], rtol=2e-6)


@pytest.mark.parametrize("lengths,single", CASES)
def test_gradients(be, lengths, single, monkeypatch):
    b = clumps(list(lengths), single, len(lengths))
    monkeypatch.setenv("LETTUCE_GB300_VJP", "pairs")
    got = []
    for method in (L.ForceMethod.direct, L.ForceMethod.tree):
        be.upload(b)
        be.adjoint_forward(L.ForceParams(G=1.0, eps=EPS, theta=0.0, method=method), 1e-2, 2, 2)
        got.append(be.adjoint_backward(b.pos64() + 0.01))
    for g, w in zip(got[1][1:], got[0][1:]):
        assert np.linalg.norm(g - w) <= 1e-5 * np.linalg.norm(w)
