"""The tree's body sort where its short form can go wrong (sorted by the leading digits of the Morton
keys only, ties ordered where the bodies are gathered, redone with every digit when the tree is
deeper than that), and the build's scans at the edges of their tiles. Keys, permutation, nodes,
moments and groups equal the oracle's bit for bit."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from gpu_util import params, zero_v
from lettuce_simulate_physics_gb300 import scenarios as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    with L.CudaBackend(0) as b:
        yield b


def same_as_oracle(be, b):
    port = O.OracleBackend("port", 0)
    port.upload(b)
    port.compute_forces(O.TREE, 1.0, 0.01, 0.6, False)
    assert np.array_equal(be.tree_keys(), port.keys())
    assert np.array_equal(be.download().id, port.download().id)
    assert be.times().interactions == port.times()["interactions"] - len(b)
    rng, mom, geo = be.tree_nodes()
    pn = port.nodes()
    assert np.array_equal(rng, np.stack([pn[f] for f in ("lo", "hi", "first", "nchild")], 1))
    for k, f in enumerate(("cx", "cy", "cz", "m", "qxx", "qxy", "qxz", "qyy", "qyz", "qzz", "rcrit2")):
        assert np.array_equal(mom[:, k], pn[f]), f
    box, lohi = be.tree_groups()
    pg = port.groups()
    assert np.array_equal(lohi, np.stack([pg["lo"], pg["hi"]], 1))


# Around the tiles of the sort (2048 bodies), the leaves (1024) and the nodes (256, 1024).
@pytest.mark.parametrize("n", [1, 2, 17, 255, 257, 1023, 1024, 1025, 2047, 2048, 2049, 4097, 33000])
def test_sizes(be, n):
    b = zero_v(S.cube(n, 11))
    be.upload(b)
    be.compute_forces(params(1, 0.01), False)
    same_as_oracle(be, b)


# Clumps of `size` bodies far closer than the sorted digits resolve: up to 16 they tie in the sort
# and are ordered by their whole keys, more make the tree deeper and the sort is redone. Every third
# clump is of coincident bodies (equal keys: the order of input).
@pytest.mark.parametrize("size", [2, 3, 15, 16, 17, 40])
@pytest.mark.parametrize("spread", [2e-6, 3e-5])
def test_ties(be, size, spread):
    rng = np.random.Generator(np.random.PCG64(size))
    c = rng.uniform(-1, 1, (300, 3))
    p = np.repeat(c, size, axis=0) + spread * rng.uniform(-1, 1, (300 * size, 3))
    for k in range(0, 300, 3):
        p[k * size:(k + 1) * size] = c[k]
    p = p[rng.permutation(len(p))]
    z = np.zeros(len(p))
    b = L.Bodies(*p.T, z, z, z, np.full(len(p), 1.0 / len(p)), np.arange(len(p)))
    be.upload(b)
    be.compute_forces(params(1, 0.01), False)
    same_as_oracle(be, b)


# A later step needs more digits than the steps before it: the bodies fall onto a few points. The
# state after it equals a fresh engine's on the same positions.
def test_deeper_later(be):
    rng = np.random.Generator(np.random.PCG64(5))
    n = 6000
    b = S.cube(n, 3)
    goal = rng.uniform(-1, 1, (20, 3))[rng.integers(0, 20, n)] + 1e-4 * rng.uniform(-1, 1, (n, 3))
    for k, f in enumerate("xyz"):
        setattr(b, "v" + f, (goal[:, k] - getattr(b, f)).astype(np.float32))
    be.upload(b)
    p = params(1, 0.01)
    be.compute_forces(p, False)
    before = be.tree_counts()["max_depth"]
    be.drift(1.0)
    now, pos = be.download(), be.pos64()
    be.compute_forces(p, False)
    assert be.tree_counts()["max_depth"] > before + 2
    a, keys, ids = be.accel(), be.tree_keys(), be.download().id
    with L.CudaBackend(0) as other:
        other.upload64(now, pos.T)
        other.compute_forces(p, False)
        assert np.array_equal(other.tree_keys(), keys) and np.array_equal(other.download().id, ids)
        assert np.array_equal(other.accel(), a)


# The moments on both sides of the leaf counts and depth widths at which they are formed by more lanes
# or in other launches (about 6 bodies a leaf: 4096 leaves, 512 and 32 768 nodes), the second call with
# the sizes of the first; a corner of the cube holds no mass (the centre is the cell's).
@pytest.mark.parametrize("n", [3000, 12000, 20000, 25000, 27000, 31000, 60000, 110000, 160000])
def test_moment_widths(be, n):
    b = zero_v(S.cube(n, n))
    b.m[(b.x < 0) & (b.y < 0) & (b.z < 0)] = 0.0
    be.upload(b)
    for _ in range(2):
        be.compute_forces(params(1, 0.01), False)
        same_as_oracle(be, b)
