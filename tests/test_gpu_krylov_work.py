"""How much an eigensolve computes when it ends early, by the kernels it launches: a start vector that is an
eigenvector already, and start vectors that are refused, cost a few products whatever krylovdim is."""
import numpy as np
import pytest

import mps_gb300 as mg
from tests.test_gpu_krylov import chain_operator

pytestmark = pytest.mark.gpu


def launches(ctx, f):
    a = ctx.counters()[0]
    r = f()
    return ctx.counters()[0] - a, r


@pytest.mark.parametrize("chi", [4, 20])
@pytest.mark.parametrize("kd", [4, 32])
def test_breakdown_and_refused_starts_cost_a_few_products(chi, kd):
    v, *ops = chain_operator(chi)
    e, x, info = mg.eigsolve_heff2(v, *ops, krylovdim=20, maxiter=200, tol=1e-11)
    op = mg.Heff2(v, *ops, precision=0)
    op(x)
    one, _ = launches(x.ctx, lambda: op(x))
    # the start's normalisation and the result's, and a product and a step each for the first one
    # and the two that may be under way when the host learns of its remainder
    most = 3 * (one + 1) + 4
    n, (e2, x2, info2) = launches(x.ctx, lambda: mg.eigsolve_heff2(x, *ops, krylovdim=kd, maxiter=8,
                                                                  tol=1e-7))
    assert info2.converged and info2.numops == 1
    np.testing.assert_allclose(e2, e, rtol=1e-9)
    assert n <= most
    for bad in (np.zeros(x.numel()), np.full(x.numel(), np.nan)):
        b = mg.from_flat(x.charge, x.space, bad)

        def refused():
            with pytest.raises(mg.MPSGError, match="zero start vector"):
                mg.eigsolve_heff2(b, *ops, krylovdim=kd, maxiter=8, tol=1e-6)
        assert launches(x.ctx, refused)[0] <= most
    np.testing.assert_allclose(mg.eigsolve_heff2(v, *ops, krylovdim=20, maxiter=200, tol=1e-11)[0], e,
                               rtol=1e-12)
