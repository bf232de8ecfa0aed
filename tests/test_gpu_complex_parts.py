"""Complex contractions (all products of the real and imaginary parts in one set of launches) against
their blocks in extended precision.

A chain of K FMAs is within K 2^-53 sum |a| |b| of its value, a product on the tensor cores (rounded
once, operands to 2^-62 of their row's largest) well within that for normal data; combining two
products adds 2 2^-53 of them. So every element is within (K + 2) 2^-53 of the sum of |a| |b| over the
products that it is made of.
"""
import numpy as np
import pytest

import mps_gb300 as mg

pytestmark = pytest.mark.gpu

# sector sizes (rows, columns, contracted): element kernel, thin kernel with either long axis, tensor
# cores, and thin and tiled sectors in one launch
SHAPES = [((1, 5), (3, 2), (1, 7)), ((33, 70), (31, 9), (40, 130)), ((5000, 9001), (4, 9), (3, 31)),
          ((4, 9), (9001, 5000), (3, 31)), ((300, 129), (81, 200), (150, 33)),
          ((5000, 300), (4, 100), (3, 200)), ((7, 300), (3, 200), (1, 5))]


def parts(shapes, rng, special):
    """Real and imaginary blocks (rows x columns per charge) of one operand."""
    out = []
    for _ in range(2):
        blocks = [rng.standard_normal(x) for x in shapes]
        if special:
            for x, v in ((blocks[0], np.inf), (blocks[1], 1e-200), (blocks[1], -0.0)):
                x[tuple(rng.integers(n) for n in x.shape)] = v
        out.append(blocks)
    return out


def flat(spaces, blocks):
    return mg.from_flat(0, spaces, np.concatenate([x.ravel(order="F") for x in blocks]))


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("imag", ["a", "b", "ab"])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_all_parts_at_once(shape, imag, special):
    rng = np.random.default_rng(31 + shape)
    ms, ns, ks = SHAPES[shape]
    V, N, K = (mg.U1Space(*enumerate(x)) for x in (ms, ns, ks))
    A = parts(list(zip(ms, ks)), rng, special)
    B = parts(list(zip(ks, ns)), rng, special)
    # contracted leg first and last, so neither operand is a fused matrix already
    at = [flat((mg.dual(K), V), [x.T for x in X]) for X in A]
    bt = [flat((mg.dual(N), K), [x.T for x in X]) for X in B[::-1]][::-1]  # either address order
    for sa, sb in ((1.0, 1.0), (-1.0, 1.0), (1.0, -1.0)):
        re, im = mg.contract_complex(at[0], at[1] if "a" in imag else None, sa, (-1, 1),
                                     bt[0], bt[1] if "b" in imag else None, sb, (2, -1),
                                     precision=0)
        ca, cb = ("a" in imag) * sa, ("b" in imag) * sb
        re, im = re.to_flat(), im.to_flat()
        p = 0
        for q, (m, n, k) in enumerate(zip(ms, ns, ks)):
            (ar, ai), (br, bi) = ([X[0][q], X[1][q]] for X in (A, B))
            for got, terms in ((re, [(1.0, ar, br), (-ca * cb, ai, bi)]),
                               (im, [(cb, ar, bi), (ca, ai, br)])):
                terms = [(c, x, y) for c, x, y in terms if c]
                with np.errstate(invalid="ignore"):
                    w = sum(c * (x.astype(np.longdouble) @ y.astype(np.longdouble))
                            for c, x, y in terms)
                    bound = (k + 2) * 2.0 ** -53 * sum(np.abs(x) @ np.abs(y) for _, x, y in terms)
                    g = got[p:p + m * n].reshape((m, n), order="F")
                    ok = np.isfinite(w)
                    assert np.array_equal(np.isnan(g), np.isnan(w))
                    assert np.array_equal(g[np.isinf(w)], w[np.isinf(w)].astype(float))
                    assert np.all(np.abs(g - w)[ok] <= bound[ok])
            p += m * n
