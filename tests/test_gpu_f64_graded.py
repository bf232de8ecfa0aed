"""FP64 products whose operands' elements differ by many orders of magnitude, element by element
against extended precision: no output may be further off than FP64 arithmetic allows, whatever
path its tile takes (seven digits, nine digits, FP64 FMAs).

Bounds, with u = 2^-53, RR the product of the powers of two above the row's and the column's largest
element, S = sum |a b| and n the number of k at which both elements are surely large (2^-5 of the row's
power of two): rounding the result 1.07 u |y|, and what is left out,
  K 2^-58.4 RR   with 28 products of digits (n >= 25 and n >= 3.24 sqrt(K) only),
  K 2^-60.9 RR   with 34 (n >= 4 and n >= sqrt(K) / 6 only),
  K 2^-74 RR     with 45, for |y| >= 2^-20 RR; (K / 32 + 6) u S for the others, which are sums of FP64 FMAs
                 or shown to be no further off."""
import numpy as np
import pytest

import mps_gb300 as mg

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def above(x):
    """The power of two above the largest |x| of each row."""
    return np.ldexp(1.0, np.frexp(np.abs(x).max(axis=1))[1])


def check(got, a, b):
    """got = a b within the bounds above, and at most (K + 2) u S off whatever the path, as FMAs are."""
    A, B = a.astype(np.longdouble), b.astype(np.longdouble)
    want, S = A @ B, np.abs(A) @ np.abs(B)
    K = a.shape[1]
    RR = np.outer(above(a), above(b.T)).astype(np.longdouble)
    n = (np.abs(a) >= above(a)[:, None] / 32).sum(1)[:, None] + (np.abs(b) >= above(b.T) / 32).sum(0) - K
    left = np.where(np.abs(want) >= 2.0 ** -20 * RR * (1 + 1e-3), K * 2.0 ** -74 * RR,
                    (K / 32 + 6) * U * S)
    left = np.maximum(left, np.where((n >= 4) & (36 * n * n >= K), K * 2.0 ** -60.9 * RR, 0))
    left = np.maximum(left, np.where((n >= 25) & (2 * n * n >= 21 * K), K * 2.0 ** -58.4 * RR, 0))
    err = np.abs(got.astype(np.longdouble) - want)
    assert np.all(err <= 1.07 * U * np.abs(want) + left), float((err / np.where(S > 0, S, 1)).max())
    assert np.all(err <= (K + 2) * U * S)


def falling(rng, m, n, k, decades):
    """Rows of a fall along k, columns of b rise: every term of a sum has the same size."""
    g = 10.0 ** (-decades * np.arange(k) / k)
    return (1 + rng.random((m, k))) * g, (1 + rng.random((k, n))) / g[:, None]


def wild(rng, m, n, k, decades):
    """Every element has a size of its own, a third are zero."""
    x = lambda *s: (rng.standard_normal(s) * 10.0 ** -rng.uniform(0, decades, s) * (rng.random(s) < 0.66))
    return x(m, k), x(k, n)


def meets_zero(rng, m, n, k, decades):
    """The large elements of a meet zeros of b."""
    a = 10.0 ** (-decades * np.arange(k) / k) * rng.choice([-1.0, 1.0], (m, k))
    b = rng.standard_normal((k, n))
    b[: k - 3] = 0.0
    return a, b


def middle(rng, m, n, k, decades):
    """Only the third digits meet: sums of exact products 2^-36 below RR."""
    a, b = (rng.integers(1, 200, s) * 2.0 ** -25 for s in ((m, k), (k, n)))
    a[:, 0], b[0] = 1.0, 0.0
    a[:, 1], b[1] = 0.0, 1.0
    return a, b


def plain(rng, m, n, k, decades):
    return rng.standard_normal((m, k)), rng.standard_normal((k, n))


CASES = [(falling, d) for d in (0, 4, 8, 12, 16, 30)] + [(wild, 6), (wild, 20), (wild, 100),
                                                        (meets_zero, 18), (middle, 0), (plain, 0)]


@pytest.mark.parametrize("make,decades", CASES)
@pytest.mark.parametrize("m,n,k", [(40, 33, 64), (64, 64, 33), (33, 64, 1031), (35, 40, 8100)])
def test_fused(make, decades, m, n, k):
    a, b = make(np.random.default_rng(5), m, n, k, decades)
    V, Kk, N = (mg.U1Space((0, d)) for d in (m, k, n))
    A = mg.from_flat(0, (V, mg.dual(Kk)), a.ravel(order="F"))
    B = mg.from_flat(0, (Kk, mg.dual(N)), b.ravel(order="F"))
    check(mg.matmul(A, B, precision=0).to_flat().reshape((m, n), order="F"), a, b)


@pytest.mark.parametrize("make,decades", CASES)
@pytest.mark.parametrize("complex_", [False, True])
def test_mapped(make, decades, complex_):
    """Operands read in place: legs (m, k1, k2) and (k2, n, k1), k1 k2 = 300."""
    m, n, k1, k2 = 40, 37, 20, 15
    rng = np.random.default_rng(6)
    parts = [make(rng, m, n, k1 * k2, decades) for _ in range(2 if complex_ else 1)]
    sp = lambda d: mg.U1Space((0, d))
    As = [mg.from_flat(0, (sp(m), sp(k1), mg.dual(sp(k2))),
                       a.reshape((m, k1, k2), order="F").ravel(order="F")) for a, _ in parts]
    Bs = [mg.from_flat(0, (sp(k2), mg.dual(sp(n)), mg.dual(sp(k1))),
                       b.reshape((k1, k2, n), order="F").transpose(1, 2, 0).ravel(order="F"))
          for _, b in parts]
    ia, ib = (1, -1, -2), (-2, 2, -1)
    if not complex_:
        got = mg.contract(As[0], ia, Bs[0], ib, precision=0).to_flat().reshape((m, n), order="F")
        check(got, *parts[0])
        return
    re, im = mg.contract_complex(As[0], As[1], 1.0, ia, Bs[0], None, 1.0, ib, precision=0)
    for got, a in ((re, parts[0][0]), (im, parts[1][0])):
        check(got.to_flat().reshape((m, n), order="F"), a, parts[0][1])
