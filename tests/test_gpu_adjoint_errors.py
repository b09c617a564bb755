"""The adjoint passes report the device's error word, and nothing but it."""
import numpy as np
import pytest

import lettuce_simulate_physics_gb300 as L
from lettuce_simulate_physics_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from lettuce_simulate_physics_gb300 import build as B
    B.build()
    with L.CudaBackend(0) as b:
        yield b


def problem(n, method):
    b = S.plummer(n, 5, cut=10)
    b.id[:] = np.arange(n)
    return b, L.ForceParams(G=1.0, eps=0.02, theta=0.6, method=method), b.pos64() + 0.01


# The low word of the total mass, 1 + 2^-52, is the bit of a wait that ran out. The diagnostics leave it
# where the host reads the error word.
@pytest.mark.parametrize("method", [0, 1])
def test_other_results_are_no_errors(be, method):
    b, p, target = problem(300, L.ForceMethod(method))
    b.m[:] = 0.0
    b.m[:2] = 1.0, 2.0 ** -52
    be.upload(b)
    be.diagnostics()
    be.adjoint_forward(p, 1e-3, 3, 2)
    be.diagnostics()
    assert np.isfinite(be.adjoint_backward(target)[0])


@pytest.mark.parametrize("n", [300, 3000])
def test_direct_passes_report_waits_that_ran_out(be, n):
    b, p, target = problem(n, L.ForceMethod.direct)
    be.upload(b)
    be.probe_wait_pending(2048)
    with pytest.raises(RuntimeError, match="device wait timed out"):
        be.adjoint_forward(p, 1e-3, 3, 2)
    be.upload(b)
    be.adjoint_forward(p, 1e-3, 3, 2)
    be.probe_wait_pending(2048)
    with pytest.raises(RuntimeError, match="device wait timed out"):
        be.adjoint_backward(target)
    be.upload(b)
    be.adjoint_forward(p, 1e-3, 3, 2)
    assert np.isfinite(be.adjoint_backward(target)[0])
    with pytest.raises(ValueError):
        be.probe_wait_pending(0)


# The gradients' arrays are the caller's until the pass has succeeded, new ones without pages among them
# (131 072 bodies: 8 MB and more).
@pytest.mark.parametrize("n", [3000, 131072])
def test_a_pass_that_fails_leaves_the_arrays_alone(be, n):
    b, p, target = problem(n, L.ForceMethod.direct)
    t = np.ascontiguousarray(target.T)
    seven = np.full((7, n), 7.0)
    d = lambda a: a.ctypes.data_as(L.backend._d)
    be.upload(b)
    be.adjoint_forward(p, 1e-3, 1, 1)
    be.probe_wait_pending(2048)
    with pytest.raises(RuntimeError, match="device wait timed out"):
        L.backend._check(be._lib.lg_adjoint_backward(be._h, *(d(t[k]) for k in range(3)), None,
                                                     *(d(seven[k]) for k in range(7))))
    assert (seven == 7.0).all()


@pytest.mark.parametrize("seeded", [False, True])
def test_a_pass_that_failed_needs_a_new_forward_pass(be, seeded):
    b, p, target = problem(500, L.ForceMethod.direct)
    backward = be.adjoint_backward_seeded if seeded else be.adjoint_backward
    be.upload(b)
    be.adjoint_forward(p, 1e-3, 3, 2)
    be.probe_wait_pending(2048)
    with pytest.raises(RuntimeError, match="device wait timed out"):
        backward(target)
    with pytest.raises(L.LogicError):
        backward(target)
    with pytest.raises(L.LogicError):
        be.kick(1e-3)
