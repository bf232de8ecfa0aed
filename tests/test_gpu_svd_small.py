"""Factorisation of small sector blocks (min dimension <= 64, one kernel for all blocks of a call)
against NumPy's SVD, block by block. Householder QR and rotations are backward stable: residual,
orthonormality and singular values within c n eps, n = 64, i.e. 1e-13 with c = 7.
"""
import numpy as np
import pytest

import mps_gb300 as mg
from oracle import symtensors as st
from oracle.symtensors import U1Space, dual_space as dual

from helpers import to_device, to_oracle

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 40), (33, 2), (3, 3), (31, 32), (32, 31), (33, 33), (63, 63), (64, 64), (63, 64),
          (64, 65), (65, 65), (256, 20), (20, 256), (257, 20), (4, 200), (64, 180), (180, 64)]


def spectra(kind, m, n, rng):
    r = min(m, n)
    U, _ = np.linalg.qr(rng.standard_normal((m, r)))
    W, _ = np.linalg.qr(rng.standard_normal((n, r)))
    if kind == "flat":
        return rng.standard_normal((m, n))
    if kind == "graded":
        return (U * 10.0 ** np.linspace(0, -20, r)) @ W.T
    if kind == "degenerate":
        return (U * np.repeat([3.0, 1e-3], [r - r // 2, r // 2])) @ W.T
    if kind == "deficient":  # rank about r / 2, zero rows and columns
        A = (U * (np.arange(r) < (r + 1) // 2)) @ W.T
        A[::3] = 0.0
        A[:, 1::4] = 0.0
        return A
    if kind == "unit":  # rows and columns of a permutation, different scales
        A = np.zeros((m, n))
        A[rng.permutation(m)[:r], rng.permutation(n)[:r]] = 10.0 ** rng.integers(-40, 1, r)
        return A
    if kind == "zero":
        return np.zeros((m, n))
    return rng.standard_normal((m, n)) * (1e-290 if kind == "tiny" else 1e+290)


@pytest.mark.parametrize("kind", ["flat", "graded", "degenerate", "deficient", "unit", "zero",
                                  "tiny", "huge"])
@pytest.mark.parametrize("method", ["exact", "gram_left"])
def test_small_blocks(kind, method):
    if method != "exact" and kind in ("zero", "tiny", "huge"):
        pytest.skip("the Gram matrix of such a block is not representable")
    rng = np.random.default_rng(7)
    V1 = U1Space(*[(c, m) for c, (m, n) in enumerate(SHAPES)])
    V2 = dual(U1Space(*[(c, n) for c, (m, n) in enumerate(SHAPES)]))
    sects, sizes = st.allsectorsandsizes(0, (V1, V2))
    A = st.SymTensor(0, (V1, V2), {s: spectra(kind, *mn, rng) for s, mn in zip(sects, sizes)})
    kept = sum(min(mn) for mn in SHAPES)
    if method == "exact":
        u, s, v = mg._svd_(to_device(A))
    else:
        u, s, v = mg.svdtrunc(to_device(A), maxdim=kept, tol=0.0, method=method)
    uo, so, vo = (to_oracle(x) for x in (u, s, v))
    for key, a in A.blocks.items():
        m, n = a.shape
        c = key[0]
        pick = lambda T: next(b for k, b in T.blocks.items() if abs(k[0]) == abs(c))
        U, S, W = pick(uo), pick(so), pick(vo)
        S = np.diag(S) if S.ndim == 2 else S
        if method != "exact" and (min(m, n) > 64 or max(m, n) > 256):
            continue  # factorised through the Gram matrix: half the digits for small values
        top = np.abs(a).max() or 1.0
        a = a / top
        np.testing.assert_allclose((U * (S / top)) @ W, a, atol=1e-13 * max(np.linalg.norm(a, 2), 1))
        np.testing.assert_allclose(U.T @ U, np.eye(len(S)), atol=1e-13)
        np.testing.assert_allclose(W @ W.T, np.eye(len(S)), atol=1e-13)
        np.testing.assert_allclose(S / top, np.linalg.svd(a, compute_uv=False),
                                   atol=1e-13 * max(np.linalg.norm(a, 2), 1))
        assert np.all(np.diff(S) <= 0)
