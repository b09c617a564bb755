"""How many passes the body sort takes: every digit once for new bodies, however they lie; afterwards the
digits that the tree at hand needs, also when it has become deeper on the way. Counted by the launches
of a force call (one per pass; the trees here have as many other launches)."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from gpu_util import params
from lettuce_simulate_physics_gb300 import scenarios as S

pytestmark = pytest.mark.gpu
N = 6000
P = params(1, 0.01)


@pytest.fixture(scope="module")
def be():
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    with L.CudaBackend(0) as b:
        yield b


def launches(be):
    before = be.launch_count()
    be.compute_forces(P, False)
    return be.launch_count() - before


def passes(be):
    return min(8, -(-3 * (be.tree_counts()["max_depth"] + 2) // 8))


def clumped(spread):
    rng = np.random.Generator(np.random.PCG64(5))
    return rng.uniform(-1, 1, (20, 3))[rng.integers(0, 20, N)] + spread * rng.uniform(-1, 1, (N, 3))


# Clumps of 300 bodies: more than a leaf's tie in the digits that a smooth scene of as many needs.
@pytest.mark.parametrize("spread", [1e-2, 1e-3, 1e-4])
def test_new_bodies_are_sorted_once(be, spread):
    be.upload(S.cube(N, 3))
    smooth = launches(be)
    z = np.zeros(N)
    be.upload(L.Bodies(*clumped(spread).T, z, z, z, np.full(N, 1.0 / N), np.arange(N)))
    assert launches(be) == smooth


@pytest.mark.parametrize("spread", [1e-2, 1e-3])
def test_deeper_trees_take_the_digits_they_need(be, spread):
    b = S.cube(N, 3)
    goal = clumped(spread)
    for k, f in enumerate("xyz"):
        setattr(b, "v" + f, (goal[:, k] - getattr(b, f)).astype(np.float32))
    be.upload(b)
    launches(be)
    shallow, few = launches(be), passes(be)
    be.drift(1.0)
    launches(be)
    deep, more = launches(be), passes(be)
    assert few < more < 8
    assert deep - shallow == more - few


# The lines of the upsweep's dispatch are drawn by what the tree has, not by what is allocated for it.
@pytest.mark.parametrize("n", [14000, 80000])
def test_headroom_changes_no_launches(n, monkeypatch):
    b = S.plummer(n, 3, cut=10)
    got = []
    for percent in (0, 25, 100):
        monkeypatch.setenv("LETTUCE_GB300_TREE_HEADROOM", str(percent))
        with L.CudaBackend(0) as be:
            be.upload(b)
            launches(be)
            got.append(launches(be) - min(8, -(-3 * (be.tree_counts()["max_depth"] + (2 if percent else 0)) // 8)))
    assert got[0] == got[1] == got[2]
