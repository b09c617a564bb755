"""Forests of more systems than one round of the upsweep's cluster kernel takes (512), with more nodes than
it takes whole trees of: every depth, the roots' among them, is formed by launches of its own. Per
system bit for bit as the plain engine."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from gpu_util import by_id, params
from lettuce_simulate_physics_gb300 import scenarios as S
from lettuce_simulate_physics_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "m", "id")


@pytest.mark.parametrize("systems", [512, 513, 700])
def test_forces(systems):
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    counts = [1 + (37 * k) % 500 for k in range(systems)]
    bs = [S.cube(c, k) for k, c in enumerate(counts)]
    for b in bs:
        b.id[:] = np.arange(len(b))
    en = Ensemble(0)
    en.upload(L.Bodies(*(np.concatenate([getattr(b, f) for b in bs]) for f in FIELDS)), counts,
              np.full(systems, 0.02), np.full(systems, 0.6), [1] * systems)
    off = np.concatenate([[0], np.cumsum(counts)])
    with L.CudaBackend(0) as be:
        for _ in range(2):  # sizes read, then those of the call before
            en.energy()
            a, ids = en.accel(), en.download().id
            for k in list(range(0, systems, 23)) + [systems - 1]:
                part = slice(off[k], off[k + 1])
                be.upload(bs[k])
                be.compute_forces(params(1, 0.02, 0.6), True)
                assert np.array_equal(by_id(ids[part], a[:, part]), by_id(be.download().id, be.accel())), k
    en.close()
