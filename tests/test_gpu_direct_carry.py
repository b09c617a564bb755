"""The sum of a split direct sum's slices where the large ones cancel: two bodies of equal mass on either
side of a massless one, in the first and the second slice, and a third 2^26 times as light in the slice
that the thread of the first one takes next. Whatever threads add the slices, the light body's pull is
what remains: three roundings of it at most (its kernel's, the product with its mass and G's)."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slices,parts", [(3, 1), (4, 2), (8, 4), (16, 8), (33, 8)])
@pytest.mark.parametrize("potential", [False, True])
def test_what_remains(slices, parts, potential, monkeypatch):
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    monkeypatch.setenv("LETTUCE_GB300_DIRECT", f"1,{slices}")
    each = 128
    n = slices * each
    x, m = np.full(n, 3.0), np.zeros(n)
    x[0] = 0.0
    for at, side, mass in ((1, 1.0, 2.0 ** 20), (each, -1.0, 2.0 ** 20), ((parts if parts > 1 else 2) * each, 1.0, 2.0 ** -6)):
        x[at], m[at] = side, mass
    z = np.zeros(n)
    with L.CudaBackend(0) as be:
        be.upload(L.Bodies(x, z, z, z, z, z, m, np.arange(n)))
        be.compute_forces(L.ForceParams(G=1.0, eps=0.5, method=L.ForceMethod.direct), potential)
        a = be.accel()[:, 0].astype(np.float64)
    # The reciprocal root's own error (2^-22.9 relative) enters three times.
    want = 2.0 ** -6 / 1.25 ** 1.5
    assert abs(a[0] - want) <= (3 * 2.0 ** -22.9 + 4 * 2.0 ** -24) * want
    assert a[1] == a[2] == 0
