"""FP64 contractions that the tensor cores do not take: no scratch for the packed operands (fused, mapped,
complex), and K beyond the digits' range. Bound: a sum of K FP64 FMAs, K 2^-53 sum |a b|."""
import numpy as np
import pytest

import mps_gb300 as mg
from mps_gb300._lib import call

pytestmark = pytest.mark.gpu


def sp(d):
    return mg.U1Space((0, d))


def check(got, a, b):
    A, B = a.astype(np.longdouble), b.astype(np.longdouble)
    err = np.abs(got.to_flat().reshape((a.shape[0], b.shape[1]), order="F") - A @ B)
    assert np.all(err <= (a.shape[1] + 2) * 2.0 ** -53 * (np.abs(A) @ np.abs(B)))


def up(x, *spaces):
    return mg.from_flat(0, spaces, x.ravel(order="F"))


@pytest.fixture
def no_scratch():
    ctx = mg.get_context()
    call("mpsg_ctx_set_scratch_limit", ctx.handle, 1 << 10)
    yield
    call("mpsg_ctx_set_scratch_limit", ctx.handle, -1)


def tiled_time_class(f):
    """The kernels of f: packing is launched by the tensor-core path only."""
    ctx = mg.get_context()
    ctx.set_timing(True)
    r = f()
    packs = ctx.kernel_time("pack")[1]
    ctx.set_timing(False)
    return r, packs


@pytest.mark.parametrize("complex_", [False, True])
def test_mapped_without_scratch(no_scratch, complex_):
    rng = np.random.default_rng(1)
    m, n, k1, k2 = 70, 45, 20, 15
    a = [rng.standard_normal((m, k1 * k2)) for _ in range(2)]
    b = rng.standard_normal((k1 * k2, n))
    As = [up(x.reshape((m, k1, k2), order="F"), sp(m), sp(k1), mg.dual(sp(k2))) for x in a]
    B = up(b.reshape((k1, k2, n), order="F").transpose(1, 2, 0), sp(k2), mg.dual(sp(n)), mg.dual(sp(k1)))
    ia, ib = (1, -1, -2), (-2, 2, -1)
    if complex_:
        (re, im), packs = tiled_time_class(lambda: mg.contract_complex(
            As[0], As[1], 1.0, ia, B, None, 1.0, ib, precision=0))
        check(re, a[0], b)
        check(im, a[1], b)
    else:
        got, packs = tiled_time_class(lambda: mg.contract(As[0], ia, B, ib, precision=0))
        check(got, a[0], b)
    assert packs == 0


def test_fused_without_scratch(no_scratch):
    rng = np.random.default_rng(2)
    a, b = rng.standard_normal((90, 130)), rng.standard_normal((130, 67))
    got, packs = tiled_time_class(lambda: mg.matmul(up(a, sp(90), mg.dual(sp(130))),
                                                    up(b, sp(130), mg.dual(sp(67))), precision=0))
    check(got, a, b)
    assert packs == 0


@pytest.mark.parametrize("k,packed", [(65536, True), (65537, False)])
def test_longest_contracted_index(k, packed):
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((33, k)), rng.standard_normal((k, 34))
    got, packs = tiled_time_class(lambda: mg.matmul(up(a, sp(33), mg.dual(sp(k))), up(b, sp(k), mg.dual(sp(34))),
                                                    precision=0))
    assert (packs > 0) == packed
    check(got, a, b)
    A = up(a.reshape((33, k, 1), order="F"), sp(33), mg.dual(sp(k)), sp(1))  # the same through index maps
    got, packs = tiled_time_class(lambda: mg.contract(A, (1, -1, 3), up(b, sp(k), mg.dual(sp(34))), (-1, 2),
                                                      precision=0))
    assert (packs > 0) == packed
    check(got, a, b)


@pytest.mark.parametrize("m,n", [(63, 127), (64, 128), (65, 129), (127, 63), (128, 64), (129, 65), (257, 33),
                                 (33, 257)])
@pytest.mark.parametrize("k", [33, 96])
def test_tile_edges(m, n, k):
    """Both sides of the 128 x 64 tile, either operand on the long one."""
    rng = np.random.default_rng(4)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    check(mg.matmul(up(a, sp(m), mg.dual(sp(k))), up(b, sp(k), mg.dual(sp(n))), precision=0), a, b)
    A = up(a.reshape((m, k, 1), order="F"), sp(m), mg.dual(sp(k)), sp(1))
    check(mg.contract(A, (1, -1, 3), up(b, sp(k), mg.dual(sp(n))), (-1, 2), precision=0), a, b)
