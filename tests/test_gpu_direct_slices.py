"""Split-j direct sums: every number of threads per body that adds the slices' partial sums (1, 2, 4, 8),
slices that do not divide evenly among them, and the default shape around the sizes where its slices
change. Against FP64."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from lettuce_simulate_physics_gb300 import scenarios as S

pytestmark = pytest.mark.gpu
EPS = 0.1


def check(n, monkeypatch, shape):
    if shape:
        monkeypatch.setenv("LETTUCE_GB300_DIRECT", shape)
    b = S.cube(n, n)
    with L.CudaBackend(0) as be:
        be.upload(b)
        be.compute_forces(L.ForceParams(G=1.0, eps=EPS, method=L.ForceMethod.direct), True)
        got = be.accel().astype(np.float64)
    x, m = b.pos64(), b.m.astype(np.float64)
    d = x[None] - x[:, None]
    s = np.sqrt((d ** 2).sum(-1) + EPS ** 2)
    a = (m[None, :, None] * d / s[..., None] ** 3).sum(1)
    phi = -(m[None] / s * (1 - np.eye(n))).sum(1)
    # Coordinates relative to a body, rounded: 2^-24 of up to twice the extent, both bodies'; d K / d x
    # is at most 3 / s^3. Then some 16 roundings per pair and in the sums.
    u = 2.0 ** -24
    move = 2 * u * 2 * np.abs(x).max() * np.sqrt(3)
    tol = (m[None] * (3 * move / s ** 3 + 16 * u * np.linalg.norm(d, axis=-1) / s ** 3)).sum(1)
    tolp = (m[None] * (move / s ** 2 + 16 * u / s)).sum(1)
    assert (np.abs(got[:3].T - a) <= tol[:, None]).all()
    assert (np.abs(got[3] - phi) <= tolp).all()


@pytest.mark.parametrize("slices", [2, 3, 4, 7, 8, 15, 16, 17, 31, 32, 39])
@pytest.mark.parametrize("n", [129, 1001])
def test_forced_slices(n, slices, monkeypatch):
    check(n, monkeypatch, f"1,{slices}")


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 300, 1023, 1024, 1025, 2047, 2048])
def test_default_shape(n, monkeypatch):
    check(n, monkeypatch, None)
