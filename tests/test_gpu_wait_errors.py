"""A bounded wait that expired in a kernel reaches the caller: the next call that returns values to the
host raises, whatever that call is, and the context works on afterwards. The record is made by a kernel
of its own (no wait is made to expire)."""
import numpy as np
import pytest

import mps_gb300 as mg
from mps_gb300 import dmrg as gd
from mps_gb300._lib import call

pytestmark = pytest.mark.gpu

ERR_CUDA = 3


def problem():
    return gd.heff_problem(64, 0.5, 1911, ncharges=9)


def svd_input():
    V, W = mg.U1Space((0, 6), (1, 5)), mg.dual(mg.U1Space((0, 6), (1, 5)))
    n = 6 * 6 + 5 * 5
    return mg.from_flat(0, (V, W), np.random.default_rng(1).standard_normal(n))


def async_copy(p):
    mg.download_async(p[0], mg.HostBuffer(p[0].numel())).synchronize()


CALLS = {
    "synchronize": lambda p: call("mpsg_ctx_synchronize", p[0].ctx.handle),
    "download": lambda p: p[0].to_flat(),
    "asynchronous copy": async_copy,
    "dot": lambda p: mg.dot(p[0], p[0]),
    "scalar contraction": lambda p: mg.contract(p[0], (-1, -2, -3, -4), mg.dual(p[0]), (-1, -2, -3, -4)),
    "svd": lambda p: mg.svdtrunc(svd_input(), maxdim=20, tol=0.0),
    "eigsolve": lambda p: mg.eigsolve_heff2(*p, krylovdim=3, maxiter=1, tol=1e-8),
}


@pytest.mark.parametrize("name", list(CALLS))
@pytest.mark.parametrize("which,text", [(0, "tensor-core GEMM"), (1, "eigsolve")])
def test_expired_wait_is_raised(name, which, text):
    p = problem()
    CALLS[name](p)
    call("mpsg_ctx_record_wait", p[0].ctx.handle, which, 3)
    with pytest.raises(mg.MPSGError, match=text) as e:
        CALLS[name](p)
    assert e.value.code == ERR_CUDA
    CALLS[name](p)  # cleared, and the context goes on
