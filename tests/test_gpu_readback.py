"""Readbacks: columns in one copy or each in its own (arrays that follow one another or not), arrays
large enough that several threads map their pages, an ensemble's systems back in the caller's
order, gradients of bodies that are not numbered in order. All exact."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from lettuce_simulate_physics_gb300 import scenarios as S
from lettuce_simulate_physics_gb300.backend import PinnedBodies
from lettuce_simulate_physics_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "m", "id")


@pytest.fixture(scope="module")
def be():
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    with L.CudaBackend(0) as b:
        yield b


def bodies(n, seed=1):
    rng = np.random.Generator(np.random.PCG64(seed))
    f = [rng.normal(size=n).astype(np.float32) for _ in range(7)]
    f[6] = np.abs(f[6]) + np.float32(0.1)
    return L.Bodies(*f, rng.permutation(n).astype(np.uint32))


@pytest.mark.parametrize("n", [1, 2, 1000, 100003, 2100000])
def test_download_gives_back_what_was_uploaded(be, n):
    b = bodies(n)
    be.upload(b)
    pinned = PinnedBodies(n)
    apart = L.Bodies.empty(n)
    for out in (be.download(), be.download(pinned.bodies), be.download(apart)):
        for f in FIELDS:
            assert np.array_equal(getattr(out, f), getattr(b, f)), f
    pinned.free()


def test_ensemble_systems_come_back_in_the_callers_order(be):
    # Direct and tree systems in turn (kept apart inside), and two without bodies.
    counts = [300, 2000, 0, 1, 1500, 700, 0]
    method = [L.ForceMethod.direct, L.ForceMethod.tree] * 3 + [L.ForceMethod.direct]
    bs = [S.plummer(max(c, 1), 40 + k, cut=10) for k, c in enumerate(counts)]
    cols = {f: np.concatenate([getattr(b, f)[:c] for b, c in zip(bs, counts)]) for f in FIELDS}
    en = Ensemble(0)
    en.upload(L.Bodies(*[cols[f] for f in FIELDS]), counts, np.full(len(counts), 0.02), np.full(len(counts), 0.6), method)
    out = en.download()
    for f in FIELDS:
        assert np.array_equal(getattr(out, f), cols[f]), f
    en.run(1e-3, 2)
    out = en.download()
    for k, c in enumerate(counts):
        part = slice(sum(counts[:k]), sum(counts[:k + 1]))
        order = np.argsort(out.id[part], kind="stable")
        assert np.array_equal(out.id[part][order], np.sort(cols["id"][part])), k
        assert np.array_equal(out.m[part][order], cols["m"][part][np.argsort(cols["id"][part], kind="stable")]), k
    en.close()


def test_gradients_of_bodies_numbered_out_of_order(be):
    n = 700
    b = S.plummer(n, 5, cut=10)
    b.id[:] = np.arange(n)
    perm = np.random.Generator(np.random.PCG64(7)).permutation(n).astype(np.uint32)
    target = b.pos64() + 0.01
    p = L.ForceParams(G=1.0, eps=0.02, method=L.ForceMethod.direct)
    be.upload(b)
    be.adjoint_forward(p, 1e-3, 4, 2)
    want = be.adjoint_backward(target)
    b.id[:] = perm
    moved = np.empty_like(target)
    moved[perm] = target
    be.upload(b)
    be.adjoint_forward(p, 1e-3, 4, 2)
    got = be.adjoint_backward(moved)
    assert got[0] == want[0]
    for g, w in zip(got[1:], want[1:]):
        assert np.array_equal(g[perm], w)
