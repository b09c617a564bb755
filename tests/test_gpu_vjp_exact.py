"""The symmetric pairwise product's sums and their combination. Bodies at one point with unit softening:
every pair's kernel is 1, and with whole masses and weights below 2^11 the single-precision sums of up
to 2^13 bodies are exact, so the gradient, m_k sum w - w_k sum m, must be too. The weights are nearly
proportional to the masses: the two products, up to 2^33, cancel to 2^24 and less, and one rounded to
single precision is off by hundreds."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    with L.CudaBackend(0) as b:
        yield b


@pytest.mark.parametrize("n", [2, 33, 64, 511, 512, 513, 1024, 1500, 2100])
def test_combination_is_exact(be, n, monkeypatch):
    monkeypatch.setenv("LETTUCE_GB300_VJP", "symmetric")
    rng = np.random.Generator(np.random.PCG64(n))
    m = rng.integers(1024, 2040, n)
    w = m[:, None] + rng.integers(0, 8, (n, 3))
    z = np.zeros(n)
    be.upload(L.Bodies(z, z, z, z, z, z, m, np.arange(n)))
    # One step of 2: the weights of its only product are dt^2 / 2 dL/dx.
    be.adjoint_forward(L.ForceParams(G=1.0, eps=1.0, method=L.ForceMethod.direct), 2.0, 1, 1)
    gx, gv, gm = be.adjoint_backward_seeded(w / 2)
    assert np.array_equal(gx, w / 2 + (m[:, None] * w.sum(0) - w * m.sum()))
    assert np.array_equal(gv, 2 * (w / 2)) and not gm.any()
