"""The FP64 block GEMM on the tensor cores against extended-precision products, and against the
FP64-pipe kernels (which the allocation-free contraction keeps) for values outside its range."""
import numpy as np
import pytest

import mps_gb300 as mg
from mps_gb300._lib import call, i32arr

pytestmark = pytest.mark.gpu

# edges of the 128 x 64 tile, of the 32-wide K step, of the 256-wide chunk between drains, both
# orientations (few rows, few columns) and several blocks of different size in one launch
SHAPES = [((33,), (33,), (33,)), ((128,), (64,), (32,)), ((129,), (65,), (257,)),
          ((40,), (513,), (256,)), ((600,), (41,), (255,)), ((1,), (200,), (40,)),
          ((64, 7, 130), (257, 50, 40), (33, 1, 1031)), ((81,), (80,), (1025,)),
          ((40,), (33,), (8100,))]


def pair(ms, ns, ks, seed=3):
    rng = np.random.Generator(np.random.Philox(seed))
    V, K, N = (mg.U1Space(*enumerate(x)) for x in (ms, ks, ns))
    a = [rng.standard_normal((m, k)) for m, k in zip(ms, ks)]
    b = [rng.standard_normal((k, n)) for k, n in zip(ks, ns)]
    return (V, K, N), a, b


def product(spaces, a, b, pipe=False):
    V, K, N = spaces
    A = mg.from_flat(0, (V, mg.dual(K)), np.concatenate([x.ravel(order="F") for x in a]))
    B = mg.from_flat(0, (K, mg.dual(N)), np.concatenate([x.ravel(order="F") for x in b]))
    if pipe:
        C = mg.zeros(0, (V, mg.dual(N)))
        call("mpsg_contract_noalloc", A.ctx.handle, A.handle, i32arr((1, -1)), B.handle,
             i32arr((-1, 2)), C.handle)
    else:
        C = mg.matmul(A, B, precision=0)  # fused matrices: the tensor cores at every size
    f, out, p = C.to_flat(), [], 0
    for x, y in zip(a, b):
        n = x.shape[0] * y.shape[1]
        out.append(f[p:p + n].reshape((x.shape[0], y.shape[1]), order="F"))
        p += n
    return out


@pytest.mark.parametrize("ms,ns,ks", SHAPES)
def test_rounded_once(ms, ns, ks):
    """Rounding the exact sum is at most 2^-53 of it; the digits left out add below 2^-57 of the
    result's norm for normal data, so a quarter more covers both. Beyond K = 8000 one more digit
    group is summed in FP32: 2^-38 per drained sum of 64 columns against a result of 2^16."""
    spaces, a, b = pair(ms, ns, ks)
    rng = np.random.default_rng(1)
    for x, y, g in zip(a, b, product(spaces, a, b)):
        rows = np.sort(rng.choice(x.shape[0], min(x.shape[0], 24), replace=False))
        want = x[rows].astype(np.longdouble) @ y.astype(np.longdouble)
        err = np.linalg.norm((g[rows] - want).astype(float))
        tol = 1.25 * 2.0 ** -53 + (2.0 ** -52 if x.shape[1] > 8000 else 0.0)
        assert err <= tol * np.linalg.norm(want.astype(float))


@pytest.mark.parametrize("ms,ns,ks", SHAPES)
def test_integers_exact(ms, ns, ks):
    spaces, a, b = pair(ms, ns, ks)
    a, b = [np.rint(50 * x) for x in a], [np.rint(50 * x) for x in b]
    for x, y, g in zip(a, b, product(spaces, a, b)):
        assert np.array_equal(g, x @ y)


def test_values_outside_the_sliced_range():
    """NaN, infinities, subnormals and rows of extreme magnitude give what the FP64 pipe gives;
    scaled ordinary rows and columns keep their relative accuracy."""
    spaces, (a,), (b,) = pair((150,), (90,), (50,))
    a[3, 4], a[12, 7] = np.inf, np.nan
    a[9, :], a[10], a[11], a[13] = 0.0, a[10] * 1e-200, a[11] * 1e200, 5e-324
    b[2, 8], b[:, 6] = -np.inf, 0.0
    b[:, 5], b[:, 9], b[:, 10] = b[:, 5] * 1e-300, b[:, 9] * 1e250, b[:, 10] * 1e-90
    (g,), (h,) = product(spaces, [a], [b]), product(spaces, [a], [b], pipe=True)
    assert np.array_equal(np.isnan(g), np.isnan(h))
    assert np.array_equal(g[np.isinf(h)], h[np.isinf(h)])
    odd = np.zeros(g.shape, bool)
    odd[[3, 10, 11, 12, 13]], odd[:, [5, 8, 9]] = True, True
    same = odd & np.isfinite(h)
    assert np.array_equal(g[same], h[same])  # the same FMA chain
    assert np.all(g[9, np.isfinite(h[9])] == 0.0)
    rest = ~odd & np.isfinite(h)
    with np.errstate(all="ignore"):
        scale = np.abs(a).max(axis=1)[:, None] * np.abs(b).max(axis=0)[None, :]
    # K FMA roundings of at most 2^-53 of partial sums below K times the scale
    assert np.all(np.abs(g[rest] - h[rest]) <= 50 * 50 * 2.0 ** -53 * scale[rest])


def noalloc(A, ia, B, ib, spaces):
    C = mg.zeros(0, spaces)
    call("mpsg_contract_noalloc", A.ctx.handle, A.handle, i32arr(ia), B.handle, i32arr(ib),
         C.handle)
    return C.to_flat()


def test_special_values_read_in_place():
    """The same through a contraction that reads its operands in place (A stored transposed, more
    than the 2^21 FMAs that stay on the FP64 pipe)."""
    (V, K, N), (a,), (b,) = pair((150,), (120,), (130,))
    a[3, 4], a[12, 7], a[9, :], a[10], b[2, 8] = np.inf, np.nan, 0.0, a[10] * 1e-200, -np.inf
    A = mg.from_flat(0, (mg.dual(K), V), a.T.ravel(order="F"))
    B = mg.from_flat(0, (K, mg.dual(N)), b.ravel(order="F"))
    g = mg.contract(A, (-1, 1), B, (-1, 2), precision=0).to_flat().reshape((150, 120), order="F")
    h = noalloc(A, (-1, 1), B, (-1, 2), (V, mg.dual(N))).reshape((150, 120), order="F")
    assert np.array_equal(np.isnan(g), np.isnan(h))
    assert np.array_equal(g[[3, 10, 12]], h[[3, 10, 12]], equal_nan=True)
    assert np.array_equal(g[:, 8], h[:, 8], equal_nan=True)
    assert np.all(g[9, np.isfinite(h[9])] == 0.0)


# thin kernel: every register variant (K up to 4, 8, 16, 32), both long axes, a unit's last rows
@pytest.mark.parametrize("m,n,k", [(90001, 9, 3), (45003, 7, 8), (5, 60007, 9), (4001, 32, 31),
                                   (31, 3300, 32)])
def test_thin_kernel_same_fma_chain(m, n, k):
    """Sparse thin operand with exact ones, zeros of both signs and non-finite values on either side:
    skipped terms leave the FMA chain's bits as they are."""
    (V, K, N), (a,), (b,) = pair((m,), (n,), (k,))
    thin, long_ = (b, a) if m >= n else (a.T, b.T)
    rng = np.random.default_rng(4)
    thin[rng.random(thin.shape) < 0.5] = 0.0
    thin[rng.random(thin.shape) < 0.2] = 1.0
    thin[0, 0] = -0.0
    long_[5, 0], long_[70, 1], long_[200, 2], long_[300, 0] = np.inf, np.nan, -0.0, -np.inf
    A = mg.from_flat(0, (mg.dual(K), V), a.T.ravel(order="F"))
    B = mg.from_flat(0, (K, mg.dual(N)), b.ravel(order="F"))
    g = mg.contract(A, (-1, 1), B, (-1, 2), precision=0).to_flat()
    h = noalloc(A, (-1, 1), B, (-1, 2), (V, mg.dual(N)))
    assert np.array_equal(g, h, equal_nan=True)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 31, 40), (7, 200, 129), (64, 64, 64)])
def test_small_kernel_same_fma_chain(m, n, k):
    (V, K, N), (a,), (b,) = pair((m,), (n,), (k,))
    a[0, 0] = np.inf if m > 1 else a[0, 0]
    A = mg.from_flat(0, (mg.dual(K), V), a.T.ravel(order="F"))
    B = mg.from_flat(0, (K, mg.dual(N)), b.ravel(order="F"))
    g = mg.contract(A, (-1, 1), B, (-1, 2), precision=0).to_flat()
    h = noalloc(A, (-1, 1), B, (-1, 2), (V, mg.dual(N)))
    assert np.array_equal(g, h, equal_nan=True)
