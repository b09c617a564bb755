"""The force walk at the edges of its packets, passes, partitions and traversal stack, against the
FP64 direct sum.

At theta 0 every body's list is all bodies, so the tree forces are the direct sum: interaction
counts are exactly N (N - 1). Tolerance: a pair term carries a handful of FP32 roundings and the
reciprocal root's error, at most about 1e-6 of the term and of random sign over a sum: relative rms
2e-6 of the accelerations; potentials, sums of one sign, 2e-6 each."""
import os

import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from gpu_util import by_id, params, rel_rms, zero_v
from lettuce_simulate_physics_gb300 import scenarios as S
from lettuce_simulate_physics_gb300.backend import LET_NODE_DTYPE
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EPS = 0.02


def engine(group=None):
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    old = os.environ.get("LETTUCE_CUDA_GROUP")
    if group is not None:
        os.environ["LETTUCE_CUDA_GROUP"] = str(group)
    try:
        return L.CudaBackend(0)
    finally:
        os.environ.pop("LETTUCE_CUDA_GROUP", None)
        if old is not None:
            os.environ["LETTUCE_CUDA_GROUP"] = old


def check(be, b, exact, theta=0.0, pairs=None):
    be.upload(zero_v(b))
    be.compute_forces(params(1, EPS, theta), True)
    n = len(b)
    ids = be.download().id
    a = by_id(ids, be.accel())
    assert be.times().interactions == (n * (n - 1) if pairs is None else pairs)
    if n > 1:
        assert rel_rms(a[:3], exact[:3]) <= 2e-6
        np.testing.assert_allclose(a[3], exact[3], rtol=2e-6)
    else:
        assert not a.any()


# Body packets hold 768 bodies; a pass takes 128 bodies, a lane two of them.
@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 127, 128, 129, 767, 768, 769, 1535, 1537, 3001])
def test_list_lengths(n):
    b = S.cube(n, 5)
    with engine() as be:
        check(be, b, O.direct_fp64(b, 1.0, EPS))


# Groups of one body (128 partitions), of odd sizes, and of several passes.
@pytest.mark.parametrize("group", [1, 2, 5, 31, 33, 64, 65, 127, 129, 255, 257, 1024])
def test_group_sizes(group):
    b = S.plummer(2500, 3)
    with engine(group) as be:
        check(be, b, O.direct_fp64(b, 1.0, EPS))


# One leaf of coincident bodies longer than a packet, among others: its range is split. Their mutual
# offset is zero, so each adds exactly m / eps to the others' potential.
@pytest.mark.parametrize("copies", [17, 40, 768, 2000])
def test_long_ranges(copies):
    b = S.cube(900, 7)
    for f in ("x", "y", "z"):
        getattr(b, f)[:copies if copies < 900 else 0] = 0.25
    if copies >= 900:
        one = np.full(copies, 0.25, np.float32)
        z = np.zeros(copies, np.float32)
        b = b.append(L.Bodies(one, one, one, z, z, z, np.full(copies, 1e-3, np.float32),
                              np.arange(copies, dtype=np.uint32)))
    with engine() as be:
        check(be, b, O.direct_fp64(b, 1.0, EPS))


# Cells fill packets of 320 (theta small: long cell lists); counts equal the oracle's.
@pytest.mark.parametrize("theta", [0.2, 0.45, 0.9])
def test_cell_lists_count(theta):
    b = S.disk(30000, 2)
    port = O.OracleBackend("port", 0)
    port.upload(zero_v(b))
    port.compute_forces(O.TREE, 1.0, EPS, theta, False)
    want = port.times()["interactions"] - len(b)
    with engine() as be:
        be.upload(zero_v(b))
        be.compute_forces(params(1, EPS, theta), False)
        assert be.times().interactions == want
        ok, cost = be.body_costs()
        assert ok and int(cost.astype(np.float64).sum()) == want


# A remote tree whose root has more than eight children (an octree's never does): every child is
# opened, so the receiver sums all its bodies.
@pytest.mark.parametrize("kids", [1, 8, 9, 16, 17, 300])
@pytest.mark.parametrize("method", [0, 1])
def test_remote_root_with_many_children(kids, method):
    b, r = S.cube(200, 3), S.cube(2 * kids, 4)
    nodes = np.zeros(1 + kids, LET_NODE_DTYPE)
    nodes["rcrit2"] = np.float32(3e38)  # always opened
    nodes[0]["first_child"], nodes[0]["child_count"] = 1, kids
    nodes["first_child"][1:] = -1
    nodes["body_first"][1:] = 2 * np.arange(kids)
    nodes["body_count"][1:] = 2
    nodes["mass"] = 1.0
    both = b.append(r)
    exact = O.direct_fp64(both, 1.0, EPS)[:, :200]
    with engine() as be:
        p = params(method, EPS, 0.0)
        be.upload(zero_v(b))
        be.build_tree(p)
        be.compute_forces_with(p, True, [L.LetTree(nodes, r.x, r.y, r.z, r.m)])
        a = by_id(be.download().id, be.accel())
        assert be.times().interactions == 200 * 199 + 200 * 2 * kids
    assert rel_rms(a[:3], exact[:3]) <= 2e-6
    np.testing.assert_allclose(a[3], exact[3], rtol=2e-6)
