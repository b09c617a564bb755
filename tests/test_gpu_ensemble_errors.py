"""A device error of any step of an ensemble run is reported by the run, whatever steps follow it. The
error is a wait that ran out, made before the run's first step by waits that nothing satisfies."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from lettuce_simulate_physics_gb300 import scenarios as S
from lettuce_simulate_physics_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "m", "id")


def ensemble(methods):
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    bs = [S.plummer(1000 + 300 * k, k, cut=10) for k in range(len(methods))]
    en = Ensemble(0)
    en.upload(L.Bodies(*(np.concatenate([getattr(b, f) for b in bs]) for f in FIELDS)), [len(b) for b in bs],
              np.full(len(bs), 0.02), np.full(len(bs), 0.6), methods)
    return en


@pytest.mark.parametrize("methods", [[1, 1, 1], [0, 1, 0, 1], [0, 0]])
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("steps", [1, 4])
def test_run_reports_an_earlier_steps_error(methods, graph, steps):
    with ensemble(methods) as en:
        en.run(1e-4, steps, graph)
        en.probe_wait_timeout(2048)
        with pytest.raises(RuntimeError, match="wait-timeout"):
            en.run(1e-4, steps, graph)
        en.run(1e-4, steps, graph)  # reported once, and usable afterwards
        assert np.isfinite(en.download().x).all()


@pytest.mark.parametrize("call", ["run", "energy"])
def test_first_forces_report_an_error(call):
    with ensemble([1, 0]) as en:
        en.probe_wait_timeout(2048)
        with pytest.raises(RuntimeError, match="wait-timeout"):
            en.run(1e-4, 2) if call == "run" else en.energy()
        e = en.energy()[0]
        assert np.isfinite(e).all()
    with ensemble([1, 0]) as en:
        with pytest.raises(ValueError):
            en.probe_wait_timeout(0)


# After a wait that ran out the permutation and the tree may be anything: the gather leaves every body
# where it is, and nothing else of the build or the walk runs.
def test_bodies_stay_in_place_after_a_wait_that_ran_out():
    n = 5000
    b = S.plummer(n, 3, cut=10)
    b.vx[:] = b.vy[:] = b.vz[:] = 0
    b.id[:] = np.arange(n)
    with ensemble([0]) as en:
        for _ in range(2):
            en.upload(b, [n], [0.02], [0.6], [1])
            en.probe_wait_timeout(2048)
            with pytest.raises(RuntimeError, match="wait-timeout"):
                en.energy()
            out = en.download()
            for f in FIELDS:
                assert np.array_equal(getattr(out, f), getattr(b, f)), f
            en.energy()
            assert not np.array_equal(en.download().id, b.id)  # sorted
