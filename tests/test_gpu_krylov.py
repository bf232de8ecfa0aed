"""The Lanczos recurrence on the device (one cooperative launch per Krylov step) against the oracle:
every register variant of the step kernel, one block and several, restarts and breakdown."""
import numpy as np
import pytest

import mps_gb300 as mg
from mps_gb300 import dmrg
from oracle import mps as om
from oracle import symtensors as st
from tests.helpers import relerr, to_oracle

pytestmark = pytest.mark.gpu


def chain_operator(chi):
    """Two-site operator at the middle of an L = 12 Heisenberg chain and a start vector."""
    mps = dmrg.mps_from_host(dmrg.random_mps_host(12, 6, chi, seed=5))
    dmrg.center_at(mps, 1)
    Ws = dmrg.xxz_u1mpo(12, 1.0)
    env = dmrg.initialenv(mps, Ws, 1)
    A = mps.As[0]
    for l in range(1, 6):
        u, s, v = mg._svd_(mg.fuselegs(A, 1, 2))
        Q = mg.splitleg(u, 1, A.space[0:2])
        env[l] = mg.mpsupdateleft(env[l - 1], Q, Ws[l - 1])
        A = mg.contract(mg.matmul(s, v), (1, -1), mps.As[l], (-1, 2, 3))
    AA = mg.contract(A, (1, 2, -1), mps.As[6], (-1, 3, 4))
    return AA, env[5], env[8], Ws[5], Ws[6]


@pytest.mark.parametrize("chi,kd,maxiter", [(4, 2, 3), (4, 4, 5), (16, 5, 8), (20, 9, 4), (16, 20, 2),
                                            (20, 32, 2)])
def test_same_solve_as_the_oracle(chi, kd, maxiter):
    """Same operation counts; eigenvalue to 1e-10 and, as the oracle's residual and gap allow,
    eigenvector to 1e-7 of its norm (both solves stop unconverged at the same step)."""
    AA, eL, eR, W1, W2 = chain_operator(chi)
    o = [to_oracle(t) for t in (AA, eL, eR, W1, W2)]
    E0, x0, i0 = om.eigsolve_lanczos(lambda v: om.applymps2site(v, *o[1:]), o[0], krylovdim=kd,
                                     maxiter=maxiter, tol=1e-9)
    E1, x1, i1 = mg.eigsolve_heff2(AA, eL, eR, W1, W2, krylovdim=kd, maxiter=maxiter, tol=1e-9)
    assert abs(E1 - E0) <= 1e-10 * abs(E0)
    assert i1.numiter == i0.numiter and i1.numops == i0.numops
    a, b = x1.to_flat(), st.flatten(x0)
    assert relerr(a * np.sign(a @ b), b) <= 1e-7


def test_breakdown_ends_the_solve_at_its_step():
    """A start vector that is an eigenvector: one operation, no restart, the vector itself."""
    AA, eL, eR, W1, W2 = chain_operator(16)
    E, x, _ = mg.eigsolve_heff2(AA, eL, eR, W1, W2, krylovdim=20, maxiter=200, tol=1e-11)
    E1, x1, info = mg.eigsolve_heff2(x, eL, eR, W1, W2, krylovdim=20, maxiter=8, tol=1e-7)
    assert info.numops == 1 and info.numiter == 1 and info.converged
    assert abs(E1 - E) <= 1e-10 * abs(E)
    assert relerr(x1.to_flat(), x.to_flat()) <= 1e-12


def test_zero_start_vector_is_refused():
    AA, eL, eR, W1, W2 = chain_operator(4)
    with pytest.raises(mg.MPSGError):
        mg.eigsolve_heff2(mg.fill_(mg.copy(AA), 0.0), eL, eR, W1, W2)


def test_vectors_too_long_for_one_cluster():
    """The vector steps of a solve whose blocks meet at the counter (the shorter vectors above take one
    cluster), against the oracle as above."""
    mps = dmrg.mps_from_host(dmrg.random_mps_host(16, 8, 60, seed=6))
    dmrg.center_at(mps, 1)
    Ws = dmrg.xxz_u1mpo(16, 1.0)
    env = dmrg.initialenv(mps, Ws, 1)
    A = mps.As[0]
    for l in range(1, 8):
        u, s, v = mg._svd_(mg.fuselegs(A, 1, 2))
        Q = mg.splitleg(u, 1, A.space[0:2])
        env[l] = mg.mpsupdateleft(env[l - 1], Q, Ws[l - 1])
        A = mg.contract(mg.matmul(s, v), (1, -1), mps.As[l], (-1, 2, 3))
    AA = mg.contract(A, (1, 2, -1), mps.As[8], (-1, 3, 4))
    args = AA, env[7], env[10], Ws[7], Ws[8]
    assert AA.numel() > 8 * 3 * 256
    o = [to_oracle(t) for t in args]
    for kd in (3, 5):
        E0, x0, i0 = om.eigsolve_lanczos(lambda v: om.applymps2site(v, *o[1:]), o[0], krylovdim=kd,
                                         maxiter=4, tol=1e-9)
        E1, x1, i1 = mg.eigsolve_heff2(*args, krylovdim=kd, maxiter=4, tol=1e-9)
        assert abs(E1 - E0) <= 1e-10 * abs(E0)
        assert i1.numiter == i0.numiter and i1.numops == i0.numops
        a, b = x1.to_flat(), st.flatten(x0)
        assert relerr(a * np.sign(a @ b), b) <= 1e-7
